// Element assembly + static condensation (the body of doassemble,
// examples/poisson2D_HDG.jl:77-174): k_element_schur and, with kappa a field, k_element_field, several
// cells to a warp; k_element_condense, a warp per cell, for cells whose reduced system is not positive.
//
// Per cell k_element_condense
//   1. gathers the three vertices and forms J, det J, adj(J) = det J * J^-1, the weighted
//      outward normals wn_f (|wn_f| = |e_f|) and the orientation bits (src/mesh.jl:51-54);
//   2. writes the augmented local system [Me | EF | Bte] of size n x (n+m+1) into shared memory,
//      Me = [Ae -Be; Be' Ce], EF = [-Ee; Fe], Bte = [0; be], every block being a combination
//      of the packed reference matrices of tables.cpp (no per-point basis loops);
//   3. eliminates with partial pivoting (the LU of `factorize`, :160) and back-substitutes all
//      m+1 right-hand sides: X = [K_e | b_e] (:171,:173);
//   4. forms [Ate | bte] = [Ee;Fe]' X - [He | 0] through the factorised form of Ee and Fe
//      (Ee = wn_f (x) F_{f,o}, Fe = tau |e_f| F_{f,o}), with bte = -[Ee;Fe]' b_e (:172,:174).
// Outputs per cell: AB = [Ate | bte] (m x (m+1)) and KB = [K_e | b_e] (n x (m+1)), row-major.
#include <map>
#include <mutex>
#include <tuple>
#include <cstdlib>
#include "hdg_device.cuh"

namespace {

struct ElemArgs {
  const double* xy;
  const int32_t* cells;
  const uint8_t* orient;
  const double* ref;
  int ref_len, nq;
  int nc;
  CoefDev co;      // per-problem source, coefficient and tau (one problem unless batched)
  int kappa_mode;  // 0: kappa = 1, 1: per-cell array, 2: per-problem field
  const double* kcell;
  double* AB;
  double* KB;
  int* err;
  int32_t* list;  // kappa field: the cells left to the general kernel (their number, their ids); NULL: all cells
  int schur;  // 1: the Schur path (invertible reference mass, kappa constant per cell), 2: with one null function,
              // 3: kappa a field, 4: with one null function
  int he_tau; // 1: He carries tau
  int unit;   // the rows of Ate have a sum that is known (RefTables::unit)
  RefLayout L;  // offsets of the packed reference tables (tables.cpp: ref_layout)
};

// One warp per cell; EWARPS warps (cells) per CTA, picked per degree, quadrature size and mesh
// size by the launch-time autotuner below.  This is the general path (any quadrature, kappa as a
// field): the full augmented system, eliminated with partial pivoting.
template <int P, int EWARPS>
__global__ void __launch_bounds__(EWARPS * 32) k_element_condense(ElemArgs a) {
  using D = Dims<P>;
  constexpr int NW = D::NW, NT = D::NT, NV = D::NV, N = D::N, M = D::M, NC = D::NC;
  // Per-warp scratch: the augmented system [Me | EF | Bte] (row stride D::LD, solution X in
  // columns N..N+M).
  constexpr int LDW = D::LD;
  constexpr int XO = N;  // first column of X
  extern __shared__ double smem[];
  double* ref = smem;
  const int nq = a.nq;
  const RefLayout L = a.L;
  // the tables this path reads, [M .. Q], sit at the start of the packed table
  const int ref_len = a.ref_len;
  for (int i = threadIdx.x; i < ref_len; i += blockDim.x) ref[i] = a.ref[i];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wstride = N * LDW + 2 * nq + NW + N + 2;
  double* W = smem + ((ref_len + 1) & ~1) + warp * wstride;
  double* sq = W + N * LDW;  // per-warp scratch: f (or kappa^-1) at the quadrature points, be
  __syncthreads();

  const int ntodo = a.list ? a.list[0] : a.nc;
  for (int todo = blockIdx.x * EWARPS + warp; todo < ntodo; todo += gridDim.x * EWARPS) {
    const int e = a.list ? a.list[1 + todo] : todo;
    // ---- geometry (reinit!, src/ScalarFunctionSpaces.jl:101-132) -------------------------
    int nid = (lane < 3) ? a.cells[3 * e + lane] : 0;
    double px = 0.0, py = 0.0;
    if (lane < 3) {
      px = a.xy[2 * nid];
      py = a.xy[2 * nid + 1];
    }
    const double x1 = __shfl_sync(0xffffffffu, px, 0), y1 = __shfl_sync(0xffffffffu, py, 0);
    const double x2 = __shfl_sync(0xffffffffu, px, 1), y2 = __shfl_sync(0xffffffffu, py, 1);
    const double x3 = __shfl_sync(0xffffffffu, px, 2), y3 = __shfl_sync(0xffffffffu, py, 2);
    const double J00 = x2 - x1, J01 = x3 - x1, J10 = y2 - y1, J11 = y3 - y1;
    const double detJ = J00 * J11 - J01 * J10;
    if (!(detJ > 0.0) && lane == 0) atomicOr(a.err, 1);
    // adj(J) = detJ * J^-1 ; Be[(c,a),j] = sum_l adj[l][c] D_l[a][j]
    const double ad00 = J11, ad01 = -J01, ad10 = -J10, ad11 = J00;
    // weighted normals (src/shapes.jl:80-87)
    double wn[3][2] = {{-(J10 - J11), J00 - J01}, {-J11, J01}, {J10, -J00}};
    double el[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) el[f] = sqrt(wn[f][0] * wn[f][0] + wn[f][1] * wn[f][1]);
    const unsigned ob = a.orient[e];
    const int prob = a.co.cell_prob[e];
    const double tau = a.co.tau[prob];
    const int fkind = a.co.fkind[prob];
    const double* fprm = a.co.fprep + a.co.foff[prob];
    double kinv = 1.0;
    if (a.kappa_mode == 1) kinv = 1.0 / a.kcell[e];
    const double smass = kinv * detJ;
    // ---- source (and kappa field) at the volume points -----------------------------------
    for (int q = lane; q < nq; q += 32) {
      double xi = ref[L.Q + 2 * q], eta = ref[L.Q + 2 * q + 1];
      double xq = (1.0 - xi - eta) * x1 + xi * x2 + eta * x3;
      double yq = (1.0 - xi - eta) * y1 + xi * y2 + eta * y3;
      sq[q] = eval_source_prepared(fkind, fprm, xq, yq);
      if (a.kappa_mode == 2) sq[nq + q] = 1.0 / eval_field_kind(a.co.kkind[prob], a.co.kprm + a.co.koff[prob], xq, yq);
    }
    __syncwarp();
    double* be = sq + 2 * nq;
    for (int i = lane; i < NW; i += 32) {
      double s = 0.0;
      for (int q = 0; q < nq; ++q) s += ref[L.NW + i * nq + q] * sq[q];
      be[i] = s * detJ;
    }
    __syncwarp();
    // ---- augmented local system ----------------------------------------------------------
    for (int idx = lane; idx < N * NC; idx += 32) {
      const int r = idx / NC, col = idx - (idx / NC) * NC;
      double v;
      if (r < NV) {
        const int c = r / NW, ia = r - c * NW;
        const double adl0 = c ? ad01 : ad00, adl1 = c ? ad11 : ad10;
        if (col < NV) {
          const int c2 = col / NW, ib = col - c2 * NW;
          if (c2 != c) {
            v = 0.0;
          } else if (a.kappa_mode == 2) {
            double s = 0.0;
            for (int q = 0; q < nq; ++q) s += ref[L.NW + ia * nq + q] * sq[nq + q] * ref[L.N + ib * nq + q];
            v = s * detJ;
          } else {
            v = smass * ref[L.M + ia * NW + ib];
          }
        } else if (col < N) {
          const int j = col - NV;
          v = -(adl0 * ref[L.D0 + ia * NW + j] + adl1 * ref[L.D1 + ia * NW + j]);
        } else if (col < N + M) {
          const int f = (col - N) / NT, j = (col - N) - f * NT;
          const int o = (ob >> f) & 1;
          v = -wn[f][c] * ref[L.F + ((f * 2 + o) * NW + ia) * NT + j];
        } else {
          v = 0.0;
        }
      } else {
        const int ia = r - NV;
        if (col < NV) {
          const int c2 = col / NW, ib = col - c2 * NW;
          const double adl0 = c2 ? ad01 : ad00, adl1 = c2 ? ad11 : ad10;
          v = adl0 * ref[L.D0 + ib * NW + ia] + adl1 * ref[L.D1 + ib * NW + ia];
        } else if (col < N) {
          const int ib = col - NV;
          v = tau * (el[0] * ref[L.C + (0 * NW + ia) * NW + ib] + el[1] * ref[L.C + (1 * NW + ia) * NW + ib] +
                     el[2] * ref[L.C + (2 * NW + ia) * NW + ib]);
        } else if (col < N + M) {
          const int f = (col - N) / NT, j = (col - N) - f * NT;
          const int o = (ob >> f) & 1;
          v = tau * el[f] * ref[L.F + ((f * 2 + o) * NW + ia) * NT + j];
        } else {
          v = be[ia];
        }
      }
      W[r * LDW + col] = v;
    }
    __syncwarp();
    // ---- Gaussian elimination with partial pivoting --------------------------------------
    // The pivot search compares |a_ik| through its bit pattern: for non-negative IEEE doubles
    // the unsigned-integer order of the bits is the numeric order, so the search runs on the
    // integer pipe instead of the (narrow) FP64 pipe.  Ties keep the smallest row, as idamax.
    double* rinv = be + NW;  // reciprocals of the pivots, reused by the back substitution
    for (int k = 0; k < N; ++k) {
      unsigned long long best = 0ull;
      int bi = N;
      for (int i = k + lane; i < N; i += 32) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(W[i * LDW + k]) & 0x7fffffffffffffffull;
        if (v > best || (v == best && i < bi)) { best = v; bi = i; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
      }
      if (best == 0ull && lane == 0) atomicOr(a.err, 2);
      if (bi != k) {
        for (int j = k + lane; j < NC; j += 32) {
          double t = W[k * LDW + j];
          W[k * LDW + j] = W[bi * LDW + j];
          W[bi * LDW + j] = t;
        }
        __syncwarp();
      }
      const double pinv = 1.0 / W[k * LDW + k];
      if (lane == 0) rinv[k] = pinv;
      for (int i = k + 1 + lane; i < N; i += 32) W[i * LDW + k] *= pinv;
      __syncwarp();
      const int cols = NC - k - 1, rows = N - k - 1;
      for (int t = lane; t < rows * cols; t += 32) {
        const int i = k + 1 + t / cols, j = k + 1 + (t - (t / cols) * cols);
        W[i * LDW + j] -= W[i * LDW + k] * W[k * LDW + j];
      }
      __syncwarp();
    }
    // ---- back substitution on the m+1 right-hand sides -----------------------------------
    for (int k = N - 1; k >= 0; --k) {
      const double dinv = rinv[k];
      for (int j = lane; j <= M; j += 32) W[k * LDW + N + j] *= dinv;
      __syncwarp();
      for (int t = lane; t < k * (M + 1); t += 32) {
        const int i = t / (M + 1), j = t - (t / (M + 1)) * (M + 1);
        W[i * LDW + N + j] -= W[i * LDW + k] * W[k * LDW + N + j];
      }
      __syncwarp();
    }
    // ---- K_e, b_e out; Y_f = wn_f,x X_qx + wn_f,y X_qy + tau |e_f| X_u into the free columns --
    double* KB = a.KB + (size_t)e * N * (M + 1);
    for (int t = lane; t < N * (M + 1); t += 32) {
      const int r = t / (M + 1), j = t - (t / (M + 1)) * (M + 1);
      KB[t] = W[r * LDW + XO + j];
    }
    for (int t = lane; t < 3 * NW * (M + 1); t += 32) {
      const int fa = t / (M + 1), j = t - (t / (M + 1)) * (M + 1);
      const int f = fa / NW, ia = fa - f * NW;
      W[fa * LDW + j] = wn[f][0] * W[ia * LDW + XO + j] + wn[f][1] * W[(NW + ia) * LDW + XO + j] +
                       tau * el[f] * W[(NV + ia) * LDW + XO + j];
    }
    __syncwarp();
    // ---- [Ate | bte] ----------------------------------------------------------------------
    double* AB = a.AB + (size_t)e * M * (M + 1);
    for (int t = lane; t < M * (M + 1); t += 32) {
      const int row = t / (M + 1), col = t - (t / (M + 1)) * (M + 1);
      const int f = row / NT, i = row - f * NT;
      const int o = (ob >> f) & 1;
      const double* F = ref + L.F + (f * 2 + o) * NW * NT;
      double s = 0.0;
#pragma unroll
      for (int ia = 0; ia < NW; ++ia) s += F[ia * NT + i] * W[(f * NW + ia) * LDW + col];
      double v;
      if (col < M) {
        const int g = col / NT, j = col - g * NT;
        v = (g == f) ? s - (a.he_tau ? tau : 1.0) * el[f] * ref[L.H + i * NT + j] : s;
      } else {
        v = -s;
      }
      AB[t] = v;
    }
    __syncwarp();
  }
}

// Schur path with an LDL' factorisation: a reference mass matrix M that is invertible, or has one null function z (p = 2
// with the default rule), and kappa constant on each cell.  Then Ae = (det J / kappa) diag(M, M) is inverted in closed form,
// and with kf = kappa / det J the condensation needs only the nw x nw Schur complement
//   S  = C + kf sum_c B_c' M^-1 B_c = C + kf (a00 Q00 + a01 (Q01 + Q01') + a11 Q11)    (SPD)
//   R' = [R'_f] with R'_f = tau |e_f| F_{f,o} + kf (b0_f DMF0_{f,o} + b1_f DMF1_{f,o}), and be,
// where B_c = adl0_c D0 + adl1_c D1, b_l f = adj(J) row l . wn_f.  A null function adds an unknown a_c per component of q,
// q_c = kf M^+ (B_c u - Ee_c u_hat) + z a_c, and the rows z' (B_c u - Ee_c u_hat) = 0: S becomes [S Z; Z' 0] with
// Z_c = B_c' z and R' gets the rows G_c = wn_f,c z' F_{f,o}; its last two pivots are negative.  Writing S = U' D U (U unit
// upper triangular) and R~ = U'^-1 [R' | be], the condensed blocks are
//   Ate_{fi,gj} = (R~' D^-1 R~)_{fi,gj} - kf (wn_f . wn_g) (F_{f,o}' M^-1 F_{g,o'})_{ij} - [f = g] |e_f| He_ij
//   bte_{fi}    = -(R~' D^-1 R~)_{fi,be}
// (the same Ate = [Ee;Fe]' Me^-1 [-Ee;Fe] - He and bte = -[Ee;Fe]' Me^-1 [0;be] that the full
// elimination of examples/poisson2D_HDG.jl:155-174 forms, reordered), symmetric by construction, so
// every pair of columns is formed once; the entries of a face's constant are tied to the rows' sums (tie_rows).  The u rows of
// [K_e | b_e], X_u = U^-1 D^-1 R~ (and a_c), are stored;
// the q rows follow linearly from them, q = kf (adl0 M^-1 D0 u + adl1 M^-1 D1 u - sum_f wn_f M^-1
// F_f u_hat_f) + z a, and are formed at recovery (k_recover_u) or when the blocks are exported (k_expand_ke).
//
// The kernel is bound by the FP64 pipe, which issues a warp instruction in 16 clocks however few of its lanes are
// active.  So a warp takes CPW = 32 / (m + 1) cells at once, a lane per right-hand-side column: 2 cells of 16 columns at
// p = 4, 2 of 13, 3 of 10, 4 of 7 at p = 3, 2, 1.  The lane keeps its column, and the column of S of the same number, in
// registers; a row of S is broadcast through shared memory when it is final.  The pairs of columns are taken
// cyclically (a lane its own column against the one d further on, d = 0..(m+1)/2), the source's terms are spread over
// (point, part) pairs and evaluated on the integer pipe (eval_part), and the entries of S spread over all lanes.  Measured
// on 65522 cells with eight bumps as the source, one cell per warp before / this layout with FP64 exponentials / here:
// p = 4 4.31 / 2.27 / 1.60 ms, p = 3 2.30 / 1.05 / 0.86, p = 2 (before: the pivoted elimination of the 18 x 18 system)
// 2.70 / 0.59 / 0.46, p = 1 1.16 / 0.22 / 0.16 (of it the rows' sums, tie_rows: 0.01 to 0.02).
// v[f] for a face index f known only at run time, without indexing a local array (which would
// place the array in local memory)
__device__ __forceinline__ double sel3(int f, double v0, double v1, double v2) {
  return f == 0 ? v0 : (f == 1 ? v1 : v2);
}

// A constant trace is the trace of a constant u with q = 0, so every row of Ate sums over the constants of the three faces
// to (tau - 1) |e_f| int mu_i (0 where He carries tau).  As differences of products the entries miss that by some roundings,
// the same ones in cells of one shape, and 1/h^2 of them goes into the solution.  So a row's entries with the constants move by
// a third each of what it misses (between two constants by a fifth of what their rows miss, which keeps the block
// symmetric and is as good as the least change), and the one with its own face's is what the others leave.  Error of u_hat
// against extended precision, pivoted elimination / without / with: 64^2 squares of p = 2 1.3e-12 / 1.1e-12 / 3.7e-13,
// distorted with kappa within a decade, 32^2 of p = 3 6.4e-14 / 7.2e-13 / 2.6e-14, 24^2 of p = 4 9.0e-14 / 1.6e-12 / 1.0e-14; of the
// entries themselves, p = 1 3.2e-16 / 3.3e-16 / 2.9e-16, p = 2 7.9e-16 / 7.8e-16 / 7.7e-16.
// us: a cell's entries, [row][face of the constant]; the lane's row is (f, fj), the cell's first lane is lane0, its rows
// follow; every lane of the warp calls it, and on says whose rows are written.
template <int NT>
__device__ __forceinline__ void tie_rows(const double* us, int f, int fj, int lane0, bool on, bool he_tau, double tau, double el,
                                         double h0, double* __restrict__ AB) {
  constexpr int COLS = 3 * NT + 1;
  const int row = f * NT + fj, fa = (f + 1) % 3, fb = (f + 2) % 3;
  const double w0 = us[row * 3], w1 = us[row * 3 + 1], w2 = us[row * 3 + 2];
  double d = (w0 + w1) + w2, target = 0.0;  // what the row misses
  if (!he_tau && __double_as_longlong(tau) != __double_as_longlong(1.0)) {
    target = (tau - 1.0) * el * h0;
    d -= target;
  }
  double e[3];  // and the rows of the constants
#pragma unroll
  for (int g = 0; g < 3; ++g) e[g] = __shfl_sync(0xffffffffu, d, lane0 + g * NT);
  const double part = fj ? -1.0 / 3.0 : -0.2;
  const double va = fma(part, fj ? d : d + sel3(fa, e[0], e[1], e[2]), sel3(fa, w0, w1, w2));
  const double vb = fma(part, fj ? d : d + sel3(fb, e[0], e[1], e[2]), sel3(fb, w0, w1, w2));
  const double own = target - (va + vb);
  if (!on) return;
  AB[row * COLS + f * NT] = own;
  AB[row * COLS + fa * NT] = va;
  AB[row * COLS + fb * NT] = vb;
  if (fj) {
    AB[f * NT * COLS + row] = own;
    AB[fa * NT * COLS + row] = va;
    AB[fb * NT * COLS + row] = vb;
  }
}

template <int P, int NZ> struct SchurDims {
  using D = Dims<P>;
  static constexpr int NW = D::NW, NT = D::NT, M = D::M;
  static constexpr int NA = NW + 2 * NZ;          // rows of [S Z; Z' 0]
  static constexpr int COLS = M + 1;              // right-hand sides: R' and be
  static constexpr int CPW = 32 / COLS;           // cells per warp
  static constexpr int TRI = NW * (NW + 1) / 2;   // S, upper triangle by columns
  static constexpr int PARTS = P == 2 || P == 3 ? 4 : 2;  // lanes per point in the source (the fuller last round)
  static constexpr int GEO = 16;                  // per cell: tau |e_f|, kf a_lm; kf wn_f . wn_g
  static constexpr int W = NA * NA, Y = NA * COLS > TRI ? NA * COLS : TRI;
  static_assert(CPW >= 1 && NA <= COLS, "a lane per column of S");
  __host__ __device__ static constexpr int tables(int nq) {  // doubles staged per CTA
    return 6 * TRI + 18 * NW * NT + NT * NT + NW * nq + 2 * nq + 36 * NT * NT + NZ * (2 * NW + 6 * NT);
  }
  __host__ __device__ static constexpr int per_warp(int nq) { return CPW * (W + Y + GEO + NW + nq + 3 * M); }
};

template <int P, int NZ>
__global__ void __launch_bounds__(256) k_element_schur(ElemArgs a) {
  using SD = SchurDims<P, NZ>;
  constexpr int NW = SD::NW, NT = SD::NT, M = SD::M, NA = SD::NA, COLS = SD::COLS, CPW = SD::CPW, TRI = SD::TRI;
  constexpr int PARTS = SD::PARTS, GEO = SD::GEO;
  extern __shared__ double smem[];
  const int nq = a.nq;
  const RefLayout G = a.L;
  // ---- tables ------------------------------------------------------------------------------------------------
  double* tS = smem;                    // [6][TRI]: C_f, Q00, Q01 + Q01', Q11
  double* tF = tS + 6 * TRI;            // [6][NW][NT]  (f, o)
  double* tD = tF + 6 * NW * NT;        // [2][6][NW][NT]  DMF
  double* tH = tD + 12 * NW * NT;       // [NT][NT]
  double* tN = tH + NT * NT;            // [NW][nq]  N times the weights
  double* tQ = tN + NW * nq;            // [nq][2]
  double* tP = tQ + 2 * nq;             // [6][6][NT][NT]  PFF
  double* tZ = tP + 36 * NT * NT;       // [2][NW] D_l' z, [6][NT] F' z
  for (int t = threadIdx.x; t < 6 * TRI; t += blockDim.x) {
    const int k = t / TRI, e = t - k * TRI;
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    const int i = e - j * (j + 1) / 2;  // i <= j
    double v;
    if (k < 3) v = a.ref[G.C + (k * NW + i) * NW + j];
    else if (k == 3) v = a.ref[G.SQ00 + i * NW + j];
    else if (k == 4) v = a.ref[G.SQ01 + i * NW + j] + a.ref[G.SQ01 + j * NW + i];
    else v = a.ref[G.SQ11 + i * NW + j];
    tS[t] = v;
  }
  for (int t = threadIdx.x; t < 6 * NW * NT; t += blockDim.x) tF[t] = a.ref[G.F + t];
  for (int t = threadIdx.x; t < 12 * NW * NT; t += blockDim.x) tD[t] = a.ref[G.SDMF + t];
  for (int t = threadIdx.x; t < NT * NT; t += blockDim.x) tH[t] = a.ref[G.H + t];
  for (int t = threadIdx.x; t < NW * nq; t += blockDim.x) tN[t] = a.ref[G.NW + t];
  for (int t = threadIdx.x; t < 2 * nq; t += blockDim.x) tQ[t] = a.ref[G.Q + t];
  for (int t = threadIdx.x; t < 36 * NT * NT; t += blockDim.x) tP[t] = a.ref[G.PFF + t];
  if constexpr (NZ > 0) {
    for (int t = threadIdx.x; t < 2 * NW; t += blockDim.x) tZ[t] = a.ref[G.ZD + t];
    for (int t = threadIdx.x; t < 6 * NT; t += blockDim.x) tZ[2 * NW + t] = a.ref[G.ZF + t];
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* base = smem + SD::tables(nq) + warp * SD::per_warp(nq);
  const bool on_lane = lane < CPW * COLS;
  const int cl = on_lane ? lane / COLS : CPW - 1;       // cell of the warp's tile
  const int col = on_lane ? lane - cl * COLS : COLS - 1; // the idle lanes repeat the last column
  double* Wc = base + cl * SD::W;                        // final rows of [S Z; Z' 0]
  double* Yc = base + CPW * SD::W + cl * SD::Y;          // D^-1 R~ (NA x COLS); before it, S by columns
  double* geo0 = base + CPW * (SD::W + SD::Y);
  double* geo = geo0 + cl * GEO;
  double* be0 = geo0 + CPW * GEO;
  double* be = be0 + cl * NW;
  double* sq0 = be0 + CPW * NW;
  double* us = sq0 + CPW * nq + cl * 3 * M;              // Ate of each row and the constant of each face
  const int f = col < M ? col / NT : 0, fj = col < M ? col - f * NT : 0;
  const int nwarps = blockDim.x >> 5;
  __syncthreads();

  for (int e0 = (blockIdx.x * nwarps + warp) * CPW; e0 < a.nc; e0 += gridDim.x * nwarps * CPW) {
    const bool mine = on_lane && e0 + cl < a.nc;
    const int e = min(e0 + cl, a.nc - 1);
    // ---- geometry (reinit!, src/ScalarFunctionSpaces.jl:101-132) -------------------------
    const int n0 = a.cells[3 * e], n1 = a.cells[3 * e + 1], n2 = a.cells[3 * e + 2];
    const double x1 = a.xy[2 * n0], y1 = a.xy[2 * n0 + 1];
    const double J00 = a.xy[2 * n1] - x1, J01 = a.xy[2 * n2] - x1;
    const double J10 = a.xy[2 * n1 + 1] - y1, J11 = a.xy[2 * n2 + 1] - y1;
    const double detJ = J00 * J11 - J01 * J10;
    if (!(detJ > 0.0) && mine && col == 0) atomicOr(a.err, 1);
    const double ad00 = J11, ad01 = -J01, ad10 = -J10, ad11 = J00;  // adj(J) = det J J^-1
    const double wx0 = J11 - J10, wy0 = J00 - J01;                  // weighted normals, src/shapes.jl:80-87
    const double wx = sel3(f, wx0, -J11, J10), wy = sel3(f, wy0, J01, -J00);  // of this lane's face
    const double el = sqrt(wx * wx + wy * wy);
    const unsigned ob = a.orient[e];
    const int fo = 2 * f + ((ob >> f) & 1);
    const int prob = a.co.cell_prob[e];
    const double tau = a.co.tau[prob];
    const double kf = (a.kappa_mode == 1) ? a.kcell[e] / detJ : 1.0 / detJ;
    if (on_lane) {  // the cell's coefficients: the columns of a face know its edge length
      if (col < M && fj == 0) geo[f] = tau * el;
      if (col == COLS - 1) {
        geo[3] = kf * (ad00 * ad00 + ad01 * ad01);
        geo[4] = kf * (ad00 * ad10 + ad01 * ad11);
        geo[5] = kf * (ad10 * ad10 + ad11 * ad11);
      }
      if (col < 6) {  // kf wn_g . wn_h for (g, h) = (0,0), (0,1), (0,2), (1,1), (1,2), (2,2)
        const int g = col < 3 ? 0 : (col < 5 ? 1 : 2), h = col < 3 ? col : (col < 5 ? col - 2 : 2);
        geo[6 + col] = kf * (sel3(g, wx0, -J11, J10) * sel3(h, wx0, -J11, J10) +
                             sel3(g, wy0, J01, -J00) * sel3(h, wy0, J01, -J00));
      }
      if (col == 6) {
        geo[12] = x1;
        geo[13] = y1;
      }
    }
    // ---- source at the volume points, be ----------------------------------------------------
    for (int t0 = 0; t0 < CPW * nq * PARTS; t0 += 32) {
      const int t = t0 + lane;
      const int pt = t / PARTS, part = t - pt * PARTS;
      const int c = min(pt / nq, CPW - 1), q = pt < CPW * nq ? pt - c * nq : 0;
      // this point's cell, from the lanes that hold its columns
      const int src = c * COLS;
      const double X = __shfl_sync(0xffffffffu, x1, src), Yv = __shfl_sync(0xffffffffu, y1, src);
      const double A00 = __shfl_sync(0xffffffffu, J00, src), A01 = __shfl_sync(0xffffffffu, J01, src);
      const double A10 = __shfl_sync(0xffffffffu, J10, src), A11 = __shfl_sync(0xffffffffu, J11, src);
      const int pr = __shfl_sync(0xffffffffu, prob, src);
      const double xi = tQ[2 * q], eta = tQ[2 * q + 1];
      double v = 0.0;
      if (pt < CPW * nq) {
        const double xq = fma(A01, eta, fma(A00, xi, X)), yq = fma(A11, eta, fma(A10, xi, Yv));
        const double sc = a.co.fix_scale[pr];
        v = eval_part(a.co.fkfix[pr], a.co.ffix + a.co.fofix[pr], xq, yq, __double2ll_rn(xq * sc),
                      __double2ll_rn(yq * sc), part, PARTS);
      }
#pragma unroll
      for (int o = PARTS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (part == 0 && pt < CPW * nq) sq0[pt] = finish_parts(a.co.fkfix[pr], v);
    }
    __syncwarp();
    if (col < NW && on_lane) {
      double t = 0.0;
      for (int q = 0; q < nq; ++q) t += tN[col * nq + q] * sq0[cl * nq + q];
      be[col] = t * detJ;
    }
    // ---- S (upper triangle, by columns) over all lanes; the columns into registers ---------------
    for (int t = lane; t < CPW * TRI; t += 32) {
      const int c = t / TRI, k = t - c * TRI;
      const double* g = geo0 + c * GEO;
      base[CPW * SD::W + c * SD::Y + k] = g[0] * tS[k] + g[1] * tS[TRI + k] + g[2] * tS[2 * TRI + k] +
                                          g[3] * tS[3 * TRI + k] + g[4] * tS[4 * TRI + k] + g[5] * tS[5 * TRI + k];
    }
    __syncwarp();
    double s[NA], r[NA], ri[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) s[i] = 0.0;
    if (col < NW) {
#pragma unroll
      for (int i = 0; i < NW; ++i)
        if (i <= col) s[i] = Yc[col * (col + 1) / 2 + i];
    }
    if constexpr (NZ > 0) {  // Z_c = B_c' z
      if (col >= NW && col < NA) {
        const double z0 = col == NW ? ad00 : ad01, z1 = col == NW ? ad10 : ad11;
#pragma unroll
        for (int i = 0; i < NW; ++i) s[i] = z0 * tZ[i] + z1 * tZ[NW + i];
      }
    }
    if (col < M) {
      const double te = tau * el, b0 = kf * (ad00 * wx + ad01 * wy), b1 = kf * (ad10 * wx + ad11 * wy);
      const double *pF = tF + fo * NW * NT + fj, *p0 = tD + fo * NW * NT + fj, *p1 = p0 + 6 * NW * NT;
#pragma unroll
      for (int i = 0; i < NW; ++i) r[i] = te * pF[i * NT] + b0 * p0[i * NT] + b1 * p1[i * NT];
      if constexpr (NZ > 0) {
        r[NW] = wx * tZ[2 * NW + fo * NT + fj];
        r[NW + 1] = wy * tZ[2 * NW + fo * NT + fj];
      }
    } else {
#pragma unroll
      for (int i = 0; i < NA; ++i) r[i] = i < NW ? be[i] : 0.0;
    }
    __syncwarp();  // S has been read: its place becomes Y
    // ---- S = U' D U (LDL', no square roots), carrying the right-hand sides ---------------------
#pragma unroll
    for (int k = 0; k < NA; ++k) {
      if (on_lane && col >= k && col < NA) Wc[k * NA + col] = s[k];
      __syncwarp();
      const double d = Wc[k * NA + k];
      const bool fits = k < NW ? d > 0.0 : d < 0.0;
      if (!fits && mine && col == 0) atomicOr(a.err, 2);  // not definite as it must be (LAPACK PosDefException)
      const double rk = recip_cubic(d);
      ri[k] = rk;
      const double ts = s[k] * rk, tr = r[k] * rk;
      if (on_lane) Yc[k * COLS + col] = tr;
#pragma unroll
      for (int i = k + 1; i < NA; ++i) {
        const double w = Wc[k * NA + i];
        s[i] -= w * ts;
        r[i] -= w * tr;
      }
    }
    __syncwarp();
    // ---- [Ate | bte]: R~' D^-1 R~ by pairs of columns, then the face-face term and He -------------
    double* AB = a.AB + (size_t)e * M * COLS;
    const double* Hh = tH + fj * NT;
    const double he = (a.he_tau ? tau : 1.0) * el;
#pragma unroll 1
    for (int d = 0; d <= COLS / 2; ++d) {
      int o = col + d;
      if (o >= COLS) o -= COLS;
      double dot = 0.0;
#pragma unroll
      for (int k = 0; k < NA; ++k) dot += r[k] * Yc[k * COLS + o];
      const bool twice = 2 * d == COLS && col >= COLS / 2;  // that pair is the other lane's
      if (mine && !twice && !(col == M && o == M)) {
        if (col == M || o == M) {
          AB[(col == M ? o : col) * COLS + M] = -dot;
        } else {
          const int g = o / NT, gj = o - g * NT, go = 2 * g + ((ob >> g) & 1);
          const int lo = min(f, g), hi = max(f, g);
          double v = dot - geo[6 + lo + hi + (lo > 0 ? 1 : 0)] * tP[((fo * 6 + go) * NT + fj) * NT + gj];
          if (f == g) v -= he * Hh[gj];
          if (gj == 0) us[col * 3 + g] = v;
          if (fj == 0) us[o * 3 + f] = v;
          if (a.unit && (fj == 0 || gj == 0)) continue;  // tied to the rows' sums below
          AB[col * COLS + o] = v;
          if (d) AB[o * COLS + col] = v;
        }
      }
    }
    __syncwarp();
    if (a.unit) tie_rows<NT>(us, f, fj, cl * COLS, mine && col < M, a.he_tau != 0, tau, el, Hh[0], AB);
    // ---- X_u = U^-1 Y in the lane's registers; a row goes out as m+1 consecutive values -----------
    double* KB = a.KB + (size_t)e * NA * COLS + col;
#pragma unroll
    for (int k = NA - 1; k >= 0; --k) {
      double t = 0.0;
#pragma unroll
      for (int i = k + 1; i < NA; ++i) t += Wc[k * NA + i] * r[i];
      r[k] = Yc[k * COLS + col] - ri[k] * t;  // R~ is not needed below row k + 1 any more
      if (mine) KB[k * COLS] = r[k];
    }
    __syncwarp();
  }
}

// The Schur path for a kappa that varies within the cell (a field), with positive volume weights.  Ae = diag(Aw, Aw) with
// Aw = int kappa^-1 phi phi' differs from cell to cell, so the products that the tables hold for a constant kappa are formed
// here: Aw = U' D U on the range of the reference mass matrix (NR functions), the 2 NW + M columns [V'D0 | V'D1 | V'F_{f,o}]
// carried along, and the products of all their pairs in the D^-1 metric, which are D_l' Aw^-1 D_m, D_l' Aw^-1 F and
// F' Aw^-1 F.  From there the condensation is that of k_element_schur.  The q rows are stored here (they need Aw).
//
// One cell per warp at p = 2 and 3 (21 and 32 columns, a lane each), two at p = 1.  The fields' modes are spread over
// (point, part) pairs: at p = 3 and 64 modes each for f and kappa, a lane per point kept 12 of 32 lanes busy for more than
// half of the 43 us a cell took an SM.  A cell with kappa <= 0 (or not finite) at a point may have an indefinite Aw; it goes
// on the list for the pivoted kernel.  Measured on 65522 cells with 64 modes each, pivoted elimination / this layout with
// FP64 cosines / here: p = 3 18.6 / 8.2 / 4.4 ms, p = 2 13.6 / 4.6 / 2.6, p = 1 11.9 / 1.7 / 0.74.
template <int P, int NZ> struct FieldDims {
  using D = Dims<P>;
  static constexpr int NW = D::NW, NT = D::NT, M = D::M, N = D::N;
  static constexpr int NR = NW - NZ, NA = NW + 2 * NZ, COLS = M + 1;
  static constexpr int NC = 2 * NW + M;           // columns of the first elimination
  static constexpr int CPW = 32 / NC;
  static constexpr int TRI = NW * (NW + 1) / 2, TRR = NR * (NR + 1) / 2, PAIRS = NC * (NC + 1) / 2;
  static constexpr int PARTS = P == 3 ? 8 : 16;   // lanes per point
  static constexpr int GEO = 8;
  static constexpr int YA = NR * NC, WA = NR * NR, W = NA * NA, Y = NA * COLS;
  static constexpr int PR = PAIRS > 2 * NR * NW ? PAIRS : 2 * NR * NW;  // products; afterwards B_c in the D^-1 metric
  static_assert(CPW >= 1, "a lane per column");
  __host__ __device__ static constexpr int tables(int nq) {
    return 3 * TRI + 6 * NW * NT + NT * NT + NW * nq + 2 * nq + TRR * nq + 2 * NR * NW + 6 * NR * NT + NW * NR +
           NZ * (3 * NW + 6 * NT);
  }
  __host__ __device__ static constexpr int per_warp(int nq) {
    return CPW * (YA + WA + PR + W + Y + GEO + NW + 2 * nq + 3 * M);
  }
};

template <int P, int NZ>
__global__ void __launch_bounds__(256) k_element_field(ElemArgs a) {
  using FD = FieldDims<P, NZ>;
  constexpr int NW = FD::NW, NT = FD::NT, M = FD::M, N = FD::N, NR = FD::NR, NA = FD::NA, COLS = FD::COLS, NC = FD::NC;
  constexpr int CPW = FD::CPW, TRI = FD::TRI, TRR = FD::TRR, PARTS = FD::PARTS, GEO = FD::GEO;
  extern __shared__ double smem[];
  const int nq = a.nq;
  const RefLayout G = a.L;
  double* tC = smem;                   // [3][TRI]
  double* tF = tC + 3 * TRI;           // [6][NW][NT]
  double* tH = tF + 6 * NW * NT;       // [NT][NT]
  double* tN = tH + NT * NT;           // [NW][nq]
  double* tQ = tN + NW * nq;           // [nq][2]
  double* tW = tQ + 2 * nq;            // [TRR][nq]  w N_i N_j in the range basis
  double* tD = tW + TRR * nq;          // [2][NR][NW]
  double* tG = tD + 2 * NR * NW;       // [6][NR][NT]
  double* tV = tG + 6 * NR * NT;       // [NW][NR]
  double* tZ = tV + NW * NR;           // [2][NW] D_l' z, [6][NT] F' z, [NW] z
  for (int t = threadIdx.x; t < 3 * TRI; t += blockDim.x) {
    const int k = t / TRI, e = t - k * TRI;
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    tC[t] = a.ref[G.C + (k * NW + (e - j * (j + 1) / 2)) * NW + j];
  }
  auto stage = [&](double* to, int from, int n) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) to[t] = a.ref[from + t];
  };
  stage(tF, G.F, 6 * NW * NT);
  stage(tH, G.H, NT * NT);
  stage(tN, G.NW, NW * nq);
  stage(tQ, G.Q, 2 * nq);
  stage(tW, G.RW, TRR * nq);
  stage(tD, G.RD, 2 * NR * NW);
  stage(tG, G.RF, 6 * NR * NT);
  stage(tV, G.RV, NW * NR);
  if constexpr (NZ > 0) {
    stage(tZ, G.ZD, 2 * NW);
    stage(tZ + 2 * NW, G.ZF, 6 * NT);
    stage(tZ + 2 * NW + 6 * NT, G.ZV, NW);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  double* base = smem + FD::tables(nq) + warp * FD::per_warp(nq);
  // first elimination: lane = (cell, column of [D0 | D1 | F])
  const bool on1 = lane < CPW * NC;
  const int cl = on1 ? lane / NC : CPW - 1, c1 = on1 ? lane - cl * NC : NC - 1;
  double* Ya = base + cl * FD::YA;                          // D^-1 R~ of the first elimination (NR x NC)
  double* Wa = base + CPW * FD::YA + cl * FD::WA;           // its rows
  double* pr = base + CPW * (FD::YA + FD::WA) + cl * FD::PR;
  double* Wc = base + CPW * (FD::YA + FD::WA + FD::PR) + cl * FD::W;
  double* Yc = base + CPW * (FD::YA + FD::WA + FD::PR + FD::W) + cl * FD::Y;
  double* geo0 = base + CPW * (FD::YA + FD::WA + FD::PR + FD::W + FD::Y);
  double* geo = geo0 + cl * GEO;
  double* be = geo0 + CPW * GEO + cl * NW;
  double* sq0 = geo0 + CPW * (GEO + NW);                    // f at the points, then kappa^-1
  double* sk0 = sq0 + CPW * nq;
  double* us = sk0 + CPW * nq + cl * 3 * M;                 // as in k_element_schur
  // second elimination: the first COLS lanes of a cell, a right-hand side each
  const bool on2 = on1 && c1 < COLS;
  const int col = min(c1, COLS - 1);
  const int f = col < M ? col / NT : 0, fj = col < M ? col - f * NT : 0;
  auto pair_at = [](int i, int j) { return i <= j ? j * (j + 1) / 2 + i : i * (i + 1) / 2 + j; };
  __syncthreads();

  for (int e0 = (blockIdx.x * nwarps + warp) * CPW; e0 < a.nc; e0 += gridDim.x * nwarps * CPW) {
    const bool mine = on1 && e0 + cl < a.nc;
    const int e = min(e0 + cl, a.nc - 1);
    const int n0 = a.cells[3 * e], n1 = a.cells[3 * e + 1], n2 = a.cells[3 * e + 2];
    const double x1 = a.xy[2 * n0], y1 = a.xy[2 * n0 + 1];
    const double J00 = a.xy[2 * n1] - x1, J01 = a.xy[2 * n2] - x1;
    const double J10 = a.xy[2 * n1 + 1] - y1, J11 = a.xy[2 * n2 + 1] - y1;
    const double detJ = J00 * J11 - J01 * J10;
    if (!(detJ > 0.0) && mine && c1 == 0) atomicOr(a.err, 1);
    const double ad00 = J11, ad01 = -J01, ad10 = -J10, ad11 = J00;
    const double wx0 = J11 - J10, wy0 = J00 - J01;
    const double wx = sel3(f, wx0, -J11, J10), wy = sel3(f, wy0, J01, -J00);
    const double el = sqrt(wx * wx + wy * wy);
    const unsigned ob = a.orient[e];
    const int fo = 2 * f + ((ob >> f) & 1);
    const int prob = a.co.cell_prob[e];
    const double tau = a.co.tau[prob];
    if (on2) {
      if (col < M && fj == 0) geo[f] = tau * el;
      if (col == COLS - 1) {
        geo[3] = ad00 * ad00 + ad01 * ad01;
        geo[4] = ad00 * ad10 + ad01 * ad11;
        geo[5] = ad10 * ad10 + ad11 * ad11;
      }
    }
    // ---- f and kappa^-1 at the points; be -------------------------------------------------------
    bool good = true;
    for (int t0 = 0; t0 < CPW * nq * PARTS; t0 += 32) {
      const int t = t0 + lane;
      const int pt = t / PARTS, part = t - pt * PARTS;
      const bool in = pt < CPW * nq;
      const int c = min(pt / nq, CPW - 1), q = in ? pt - c * nq : 0, src = c * NC;
      const double X = __shfl_sync(0xffffffffu, x1, src), Yv = __shfl_sync(0xffffffffu, y1, src);
      const double A00 = __shfl_sync(0xffffffffu, J00, src), A01 = __shfl_sync(0xffffffffu, J01, src);
      const double A10 = __shfl_sync(0xffffffffu, J10, src), A11 = __shfl_sync(0xffffffffu, J11, src);
      const int po = __shfl_sync(0xffffffffu, prob, src);
      const double xi = tQ[2 * q], eta = tQ[2 * q + 1];
      const double xq = fma(A01, eta, fma(A00, xi, X)), yq = fma(A11, eta, fma(A10, xi, Yv));
      double v = 0.0, w = 0.0;
      if (in) {
        const double sc = a.co.fix_scale[po];
        const long long xf = __double2ll_rn(xq * sc), yf = __double2ll_rn(yq * sc);
        v = eval_part(a.co.fkfix[po], a.co.ffix + a.co.fofix[po], xq, yq, xf, yf, part, PARTS);
        w = eval_part(a.co.kkfix[po], a.co.kfix + a.co.kofix[po], xq, yq, xf, yf, part, PARTS);
      }
#pragma unroll
      for (int o = PARTS / 2; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
        w += __shfl_xor_sync(0xffffffffu, w, o);
      }
      if (part == 0 && in) {
        sq0[pt] = finish_parts(a.co.fkfix[po], v);
        w = finish_parts(a.co.kkfix[po], w);
        sk0[pt] = 1.0 / w;
        good = good && w > 0.0 && w < 1e300;
      }
    }
    const bool all_good = __all_sync(0xffffffffu, good);
    __syncwarp();
    if (!all_good) {  // the tile's cells go to the pivoted kernel
      if (mine && c1 == 0) a.list[1 + atomicAdd(a.list, 1)] = e;
      continue;
    }
    if (c1 < NW && on1) {
      double t = 0.0;
      for (int q = 0; q < nq; ++q) t += tN[c1 * nq + q] * sq0[cl * nq + q];
      be[c1] = t * detJ;
    }
    // ---- Aw / det J (upper triangle, by columns) over all lanes, into the place of the products ---
    for (int t = lane; t < CPW * TRR; t += 32) {
      const int c = t / TRR, k = t - c * TRR;
      double v = 0.0;
      for (int q = 0; q < nq; ++q) v += tW[k * nq + q] * sk0[c * nq + q];
      base[CPW * (FD::YA + FD::WA) + c * FD::PR + k] = v;
    }
    __syncwarp();
    double ra[NR];
    {
      double s[NR], g[NR];
#pragma unroll
      for (int i = 0; i < NR; ++i) s[i] = 0.0;
      if (c1 < NR) {
#pragma unroll
        for (int i = 0; i < NR; ++i)
          if (i <= c1) s[i] = pr[c1 * (c1 + 1) / 2 + i] * detJ;
      }
      {
        const int fc = c1 < 2 * NW ? 0 : c1 - 2 * NW, ff = fc / NT;
        const double* from = c1 < 2 * NW ? tD + (c1 / NW) * NR * NW + c1 % NW
                                         : tG + (2 * ff + ((ob >> ff) & 1)) * NR * NT + (fc - ff * NT);
        const int ld = c1 < 2 * NW ? NW : NT;
#pragma unroll
        for (int i = 0; i < NR; ++i) g[i] = from[i * ld];
      }
      __syncwarp();
      // ---- Aw = U' D U, carrying the columns ------------------------------------------------------
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        if (on1 && c1 >= k && c1 < NR) Wa[k * NR + c1] = s[k];
        __syncwarp();
        const double d = Wa[k * NR + k];
        if (!(d > 0.0) && mine && c1 == 0) atomicOr(a.err, 2);
        const double rk = recip_cubic(d);
        ra[k] = rk;
        const double ts = s[k] * rk, tg = g[k] * rk;
        if (on1) Ya[k * NC + c1] = tg;
#pragma unroll
        for (int i = k + 1; i < NR; ++i) {
          const double w = Wa[k * NR + i];
          s[i] -= w * ts;
          g[i] -= w * tg;
        }
      }
      __syncwarp();
      // ---- products of all pairs of columns -------------------------------------------------------
#pragma unroll 1
      for (int d = 0; d <= NC / 2; ++d) {
        int o = c1 + d;
        if (o >= NC) o -= NC;
        double dot = 0.0;
#pragma unroll
        for (int k = 0; k < NR; ++k) dot += g[k] * Ya[k * NC + o];
        if (on1 && !(2 * d == NC && c1 >= NC / 2)) pr[pair_at(c1, o)] = dot;  // at 2 d = NC: the other lane's pair
      }
    }
    __syncwarp();
    // ---- S and R' --------------------------------------------------------------------------------
    double s[NA], r[NA], ri[NA];
#pragma unroll
    for (int i = 0; i < NA; ++i) s[i] = 0.0;
    if (col < NW) {
#pragma unroll
      for (int i = 0; i < NW; ++i)
        if (i <= col) {
          const int k = col * (col + 1) / 2 + i;
          s[i] = geo[0] * tC[k] + geo[1] * tC[TRI + k] + geo[2] * tC[2 * TRI + k] + geo[3] * pr[pair_at(i, col)] +
                 geo[4] * (pr[pair_at(i, NW + col)] + pr[pair_at(col, NW + i)]) + geo[5] * pr[pair_at(NW + i, NW + col)];
        }
    }
    if constexpr (NZ > 0) {
      if (col >= NW && col < NA) {
        const double z0 = col == NW ? ad00 : ad01, z1 = col == NW ? ad10 : ad11;
#pragma unroll
        for (int i = 0; i < NW; ++i) s[i] = z0 * tZ[i] + z1 * tZ[NW + i];
      }
    }
    if (col < M) {
      const double te = tau * el, b0 = ad00 * wx + ad01 * wy, b1 = ad10 * wx + ad11 * wy;
#pragma unroll
      for (int i = 0; i < NW; ++i)
        r[i] = te * tF[(fo * NW + i) * NT + fj] + b0 * pr[pair_at(i, 2 * NW + col)] + b1 * pr[pair_at(NW + i, 2 * NW + col)];
      if constexpr (NZ > 0) {
        r[NW] = wx * tZ[2 * NW + fo * NT + fj];
        r[NW + 1] = wy * tZ[2 * NW + fo * NT + fj];
      }
    } else {
#pragma unroll
      for (int i = 0; i < NA; ++i) r[i] = i < NW ? be[i] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < NA; ++k) {
      if (on2 && col >= k && col < NA) Wc[k * NA + col] = s[k];
      __syncwarp();
      const double d = Wc[k * NA + k];
      const bool fits = k < NW ? d > 0.0 : d < 0.0;
      if (!fits && mine && c1 == 0) atomicOr(a.err, 2);
      const double rk = recip_cubic(d);
      ri[k] = rk;
      const double ts = s[k] * rk, tr = r[k] * rk;
      if (on2) Yc[k * COLS + col] = tr;
#pragma unroll
      for (int i = k + 1; i < NA; ++i) {
        const double w = Wc[k * NA + i];
        s[i] -= w * ts;
        r[i] -= w * tr;
      }
    }
    __syncwarp();
    // ---- [Ate | bte] -------------------------------------------------------------------------------
    double* AB = a.AB + (size_t)e * M * COLS;
    const double* Hh = tH + fj * NT;
    const double he = (a.he_tau ? tau : 1.0) * el;
#pragma unroll 1
    for (int d = 0; d <= COLS / 2; ++d) {
      int o = col + d;
      if (o >= COLS) o -= COLS;
      double dot = 0.0;
#pragma unroll
      for (int k = 0; k < NA; ++k) dot += r[k] * Yc[k * COLS + o];
      const bool twice = 2 * d == COLS && col >= COLS / 2;
      if (mine && on2 && !twice && !(col == M && o == M)) {
        if (col == M || o == M) {
          AB[(col == M ? o : col) * COLS + M] = -dot;
        } else {
          const int g = o / NT, gj = o - g * NT;
          const double gx = sel3(g, wx0, -J11, J10), gy = sel3(g, wy0, J01, -J00);
          double v = dot - (wx * gx + wy * gy) * pr[pair_at(2 * NW + col, 2 * NW + o)];
          if (f == g) v -= he * Hh[gj];
          if (gj == 0) us[col * 3 + g] = v;
          if (fj == 0) us[o * 3 + f] = v;
          if (a.unit && (fj == 0 || gj == 0)) continue;
          AB[col * COLS + o] = v;
          if (d) AB[o * COLS + col] = v;
        }
      }
    }
    __syncwarp();
    if (a.unit) tie_rows<NT>(us, f, fj, cl * NC, mine && on2 && col < M, a.he_tau != 0, tau, el, Hh[0], AB);
    // ---- X_u (and a_c), kept for the q rows in the place of Y -----------------------------------------
    double* KB = a.KB + (size_t)e * N * COLS;
#pragma unroll
    for (int k = NA - 1; k >= 0; --k) {
      double t = 0.0;
#pragma unroll
      for (int i = k + 1; i < NA; ++i) t += Wc[k * NA + i] * r[i];
      r[k] = Yc[k * COLS + col] - ri[k] * t;
      if (mine && on2 && k < NW) KB[(2 * NW + k) * COLS + col] = r[k];
    }
    __syncwarp();
    if (on2) {
#pragma unroll
      for (int k = 0; k < NA; ++k) Yc[k * COLS + col] = r[k];
    }
    // B_c = adl0_c D0 + adl1_c D1 in the D^-1 metric, [2][NR][NW], in the place of the products
    for (int t = c1; t < 2 * NR * NW; t += NC)
      if (on1) {
        const int c = t / (NR * NW), ki = t - c * NR * NW, k = ki / NW, i = ki - k * NW;
        pr[t] = (c ? ad01 : ad00) * Ya[k * NC + i] + (c ? ad11 : ad10) * Ya[k * NC + NW + i];
      }
    __syncwarp();
    // ---- q rows: Aw q_c = B_c u - wn_f,c F u_hat, a lane per (component, column) -----------------------
    for (int t = c1; t < 2 * COLS; t += NC) {
      const int c = t / COLS, j = t - c * COLS;
      double x[NW], v[NR];
#pragma unroll
      for (int i = 0; i < NW; ++i) x[i] = Yc[i * COLS + j];
      double wc = 0.0;
      if (j < M) {
        const int g = j / NT;
        wc = c ? sel3(g, wy0, J01, -J00) : sel3(g, wx0, -J11, J10);
      }
#pragma unroll
      for (int k = NR - 1; k >= 0; --k) {
        double u = j < M ? -wc * Ya[k * NC + 2 * NW + j] : 0.0;
#pragma unroll
        for (int i = 0; i < NW; ++i) u += pr[(c * NR + k) * NW + i] * x[i];
        double w = 0.0;
#pragma unroll
        for (int i = k + 1; i < NR; ++i) w += Wa[k * NR + i] * v[i];
        v[k] = u - ra[k] * w;
      }
      if (mine) {
#pragma unroll
        for (int ia = 0; ia < NW; ++ia) {
          double qv;
          if constexpr (NZ > 0) {
            qv = tZ[2 * NW + 6 * NT + ia] * Yc[(NW + c) * COLS + j];
#pragma unroll
            for (int k = 0; k < NR; ++k) qv += tV[ia * NR + k] * v[k];
          } else {
            qv = v[ia];
          }
          KB[(c * NW + ia) * COLS + j] = qv;
        }
      }
    }
    __syncwarp();
  }
}

// The q rows of [K_e | b_e] from the stored u rows (the Schur path stores X_u only, and a_c below it):
// X_q,c = kf (adl0_c M^-1 D0 X_u + adl1_c M^-1 D1 X_u - [j < m] wn_f,c M^-1 F_{f,o}), one thread per
// entry of the full n x (m+1) block.  Used when the blocks are exported, not on the solve path.
template <int P, int NZ>
__global__ void k_expand_ke(ElemArgs a, const double* __restrict__ KBu, double* __restrict__ KB) {
  using D = Dims<P>;
  constexpr int NW = D::NW, NT = D::NT, NV = D::NV, N = D::N, M = D::M, NA = NW + 2 * NZ;
  const RefLayout G = a.L;
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)a.nc * N * (M + 1)) return;
  const int e = (int)(t / (N * (M + 1)));
  const int rj = (int)(t - (int64_t)e * N * (M + 1));
  const int r = rj / (M + 1), j = rj - r * (M + 1);
  const double* Xu = KBu + (size_t)e * NA * (M + 1);
  if (r >= NV) {
    KB[t] = Xu[(r - NV) * (M + 1) + j];
    return;
  }
  const int n0 = a.cells[3 * e], n1 = a.cells[3 * e + 1], n2 = a.cells[3 * e + 2];
  const double J00 = a.xy[2 * n1] - a.xy[2 * n0], J01 = a.xy[2 * n2] - a.xy[2 * n0];
  const double J10 = a.xy[2 * n1 + 1] - a.xy[2 * n0 + 1], J11 = a.xy[2 * n2 + 1] - a.xy[2 * n0 + 1];
  const double detJ = J00 * J11 - J01 * J10;
  const double ad00 = J11, ad01 = -J01, ad10 = -J10, ad11 = J00;
  const double wn[3][2] = {{-(J10 - J11), J00 - J01}, {-J11, J01}, {J10, -J00}};
  const double kinv = (a.kappa_mode == 1) ? 1.0 / a.kcell[e] : 1.0;
  const double kf = 1.0 / (kinv * detJ);
  const int c = r / NW, ia = r - c * NW;
  double g0 = 0.0, g1 = 0.0;
  for (int ib = 0; ib < NW; ++ib) {
    const double x = Xu[ib * (M + 1) + j];
    g0 += a.ref[G.SMD0 + ia * NW + ib] * x;
    g1 += a.ref[G.SMD1 + ia * NW + ib] * x;
  }
  double v = c ? (ad01 * g0 + ad11 * g1) : (ad00 * g0 + ad10 * g1);
  if (j < M) {
    const int f = j / NT, jj = j - f * NT;
    const int fo = f * 2 + ((a.orient[e] >> f) & 1);
    v -= wn[f][c] * a.ref[G.SMF + (fo * NW + ia) * NT + jj];
  }
  KB[t] = kf * v + (NZ ? a.ref[G.ZV + ia] * Xu[(NW + c) * (M + 1) + j] : 0.0);
}

template <int P, int EWARPS> size_t smem_bytes_lu(const ElemArgs& a) {
  using D = Dims<P>;
  const int wstride = D::N * D::LD + 2 * a.nq + D::NW + D::N + 2;
  return (size_t)(((a.ref_len + 1) & ~1) + EWARPS * wstride) * sizeof(double);
}

constexpr size_t ELEM_SMEM_MAX = 200 * 1024;

int sm_count(int device) {
  int n = 152;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
  return n;
}

// Launches one path's kernel with `warps` warps per CTA and a grid of `oversub` x the resident CTAs
// (a grid-stride loop covers the rest).  Returns false when the configuration does not fit.
template <class K>
bool launch_kernel(hdg_system* s, cudaStream_t st, const ElemArgs& a, K kern, int warps, int cells_per_warp, size_t smem,
                   int oversub) {
  if (smem > ELEM_SMEM_MAX) return false;
  HDG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ELEM_SMEM_MAX));
  int blocks_per_sm = 0;
  HDG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, kern, warps * 32, smem));
  if (blocks_per_sm < 1) return false;
  const long per = (long)warps * cells_per_warp, need = (a.nc + per - 1) / per;
  long grid = std::min<long>(need, (long)sm_count(s->ctx->device) * blocks_per_sm * oversub);
  if (grid < 1) grid = 1;
  kern<<<(unsigned)grid, warps * 32, smem, st>>>(a);
  HDG_CUDA(cudaGetLastError());
  s->ctx->launches++;
  return true;
}

template <int P, int EWARPS> bool launch_lu(hdg_system* s, cudaStream_t st, const ElemArgs& a, int oversub) {
  return launch_kernel(s, st, a, k_element_condense<P, EWARPS>, EWARPS, 1, smem_bytes_lu<P, EWARPS>(a), oversub);
}

template <int P, int NZ> bool launch_schur(hdg_system* s, cudaStream_t st, const ElemArgs& a, int warps, int oversub) {
  using SD = SchurDims<P, NZ>;
  if (warps > 8) return false;  // the kernel's launch bound
  const size_t smem = sizeof(double) * ((size_t)SD::tables(a.nq) + (size_t)warps * SD::per_warp(a.nq));
  return launch_kernel(s, st, a, k_element_schur<P, NZ>, warps, SD::CPW, smem, oversub);
}

// The kappa-field kernel, then the pivoted one over the cells that it listed (mostly none).
template <int P, int NZ> bool launch_field(hdg_system* s, cudaStream_t st, const ElemArgs& a, int warps, int oversub) {
  using FD = FieldDims<P, NZ>;
  if (warps > 8) return false;  // the kernel's launch bound
  const size_t smem = sizeof(double) * ((size_t)FD::tables(a.nq) + (size_t)warps * FD::per_warp(a.nq));
  if (smem > ELEM_SMEM_MAX) return false;
  HDG_CUDA(cudaMemsetAsync(a.list, 0, sizeof(int32_t), st));
  ElemArgs all = a;
  if (!launch_kernel(s, st, all, k_element_field<P, NZ>, warps, FD::CPW, smem, oversub)) return false;
  return launch_lu<P, 2>(s, st, a, 1);
}

template <int P> bool launch_cfg(hdg_system* s, cudaStream_t st, const ElemArgs& a, int warps, int oversub) {
  if constexpr (P <= 3) {
    if (a.schur == 3) return launch_field<P, 0>(s, st, a, warps, oversub);
  }
  if constexpr (P == 2) {
    if (a.schur == 4) return launch_field<P, 1>(s, st, a, warps, oversub);
  }
  if (a.schur == 1) return launch_schur<P, 0>(s, st, a, warps, oversub);
  if constexpr (P == 2) {
    if (a.schur == 2) return launch_schur<P, 1>(s, st, a, warps, oversub);
  }
  switch (warps) {
    case 1: return launch_lu<P, 1>(s, st, a, oversub);
    case 2: return launch_lu<P, 2>(s, st, a, oversub);
    case 4: return launch_lu<P, 4>(s, st, a, oversub);
    case 8: return launch_lu<P, 8>(s, st, a, oversub);
    case 16: return launch_lu<P, 16>(s, st, a, oversub);
  }
  return false;
}

// Autotuner: the first launch for a (device, degree, quadrature size, log2 of the cell count, path)
// times every (warps per CTA, grid oversubscription) pair on the real inputs, on at most the first
// 65536 cells (the kernel only writes its outputs from its inputs, and every configuration
// computes each cell with the same instruction sequence, so the results are bit-identical; the
// real launch that follows writes every cell), and keeps the fastest.  The choice is cached for
// the process.  On a thread that builds one-shot systems (g_tuning_allowed false) a key without a
// cached choice takes the cached choice of the nearest cell count for the same degree, quadrature
// and path, and is timed only when there is none.  HDG_ELEMENT_WARPS=<1|2|4|8|16> fixes the warps
// per CTA instead.
template <int P> void launch_p(hdg_system* s, cudaStream_t st, const ElemArgs& a) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, int>, std::pair<int, int>> best;
  if (const char* env = std::getenv("HDG_ELEMENT_WARPS")) {
    const int w = std::atoi(env);
    if (!launch_cfg<P>(s, st, a, a.schur ? std::min(w, 8) : w, 4)) throw HdgError{HDG_ERR_ARG, "HDG_ELEMENT_WARPS does not fit"};
    return;
  }
  int lg = 0;
  while ((1L << (lg + 1)) <= (long)a.nc) ++lg;
  const auto key = std::make_tuple(s->ctx->device, a.nq, lg, a.schur);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = best.find(key);
    if (it == best.end() && !g_tuning_allowed) {  // nearest cached cell count, same degree and path
      int dist = 1 << 30;
      for (auto jt = best.begin(); jt != best.end(); ++jt) {
        const auto& k = jt->first;
        if (std::get<0>(k) != std::get<0>(key) || std::get<1>(k) != a.nq || std::get<3>(k) != a.schur) continue;
        const int d = std::abs(std::get<2>(k) - lg);
        if (d < dist) {
          dist = d;
          it = jt;
        }
      }
    }
    if (it != best.end()) {
      launch_cfg<P>(s, st, a, it->second.first, it->second.second);
      return;
    }
  }
  float best_ms = 1e30f;
  std::pair<int, int> pick{4, 4};
  cudaEvent_t e0, e1;
  HDG_CUDA(cudaEventCreate(&e0));
  HDG_CUDA(cudaEventCreate(&e1));
  ElemArgs t = a;  // the trials run on a prefix of the cells
  t.nc = std::min(a.nc, 65536);
  for (int w : {1, 2, 4, 8, 16})
    for (int g : {1, 4}) {
      if (!launch_cfg<P>(s, st, t, w, g)) continue;  // warm-up launch of this configuration
      HDG_CUDA(cudaEventRecord(e0, st));
      launch_cfg<P>(s, st, t, w, g);
      HDG_CUDA(cudaEventRecord(e1, st));
      HDG_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      HDG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best_ms) {
        best_ms = ms;
        pick = {w, g};
      }
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (best_ms == 1e30f) throw HdgError{HDG_ERR_ARG, "no element-kernel configuration fits in shared memory"};
  {
    std::lock_guard<std::mutex> lk(mu);
    best[key] = pick;
  }
  launch_cfg<P>(s, st, a, pick.first, pick.second);
}

}  // namespace

namespace {
ElemArgs element_args(hdg_system* s) {
  hdg_space* sp = s->space;
  hdg_mesh* m = sp->mesh;
  ElemArgs a;
  a.xy = m->d_xy.p;
  a.cells = m->d_cells.p;
  a.orient = m->d_orient.p;
  a.ref = sp->d_ref.p;
  a.nq = sp->t.nq;
  a.nc = m->nc;
  ensure_fixed_fields(s, true);
  a.co = s->coef_dev();
  a.kappa_mode = s->kappa_cells ? 1 : (s->kappa_field ? 2 : 0);
  a.he_tau = s->he_tau ? 1 : 0;
  a.unit = sp->t.unit ? 1 : 0;
  a.kcell = s->d_kappa.p;
  a.AB = s->d_AB.p;
  a.KB = s->d_KB.p;
  a.err = reinterpret_cast<int*>(s->d_scal.p + 1);
  // Schur path: its tables are valid (2: with a null function) and kappa is constant on each cell (a kappa field
  // makes Ae a weighted mass matrix that is no multiple of the reference one)
  a.schur = (sp->t.schur && a.kappa_mode != 2) ? 1 + sp->t.nullity : 0;
  // ... or a field: the same with Aw formed per cell, where the weights are positive (the rules of p = 4 are not)
  if (sp->t.schur && a.kappa_mode == 2 && sp->t.positive && sp->t.p <= 3) a.schur = 3 + sp->t.nullity;
  if (std::getenv("HDG_ELEMENT_FULL_LU") != nullptr) a.schur = 0;
  a.list = nullptr;
  if (a.schur >= 3) {
    s->d_elem_list.alloc((size_t)m->nc + 1);
    a.list = s->d_elem_list.p;
  }
  a.L = ref_layout(sp->t.nw, sp->t.nt, sp->t.nq);
  a.ref_len = a.L.SMD0;  // the full path stages [M .. Q]; the Schur path stages its own ranges
  return a;
}
}  // namespace

void launch_element_condense(hdg_system* s, cudaStream_t st) {
  const ElemArgs a = element_args(s);
  s->kb_u_only = a.schur == 1 || a.schur == 2;
  switch (s->space->t.p) {
    case 1: launch_p<1>(s, st, a); break;
    case 2: launch_p<2>(s, st, a); break;
    case 3: launch_p<3>(s, st, a); break;
    case 4: launch_p<4>(s, st, a); break;
    default: throw HdgError{HDG_ERR_ARG, "degree not supported"};
  }
}

void launch_expand_ke(hdg_system* s, double* out, cudaStream_t st) {
  const ElemArgs a = element_args(s);
  const int64_t tot = (int64_t)a.nc * s->n * (s->m + 1);
  const unsigned grid = (unsigned)((tot + 255) / 256);
  switch (s->space->t.p) {
    case 1: k_expand_ke<1, 0><<<grid, 256, 0, st>>>(a, s->d_KB.p, out); break;
    case 2:
      if (s->space->t.nullity) k_expand_ke<2, 1><<<grid, 256, 0, st>>>(a, s->d_KB.p, out);
      else k_expand_ke<2, 0><<<grid, 256, 0, st>>>(a, s->d_KB.p, out);
      break;
    case 3: k_expand_ke<3, 0><<<grid, 256, 0, st>>>(a, s->d_KB.p, out); break;
    case 4: k_expand_ke<4, 0><<<grid, 256, 0, st>>>(a, s->d_KB.p, out); break;
    default: throw HdgError{HDG_ERR_ARG, "degree not supported"};
  }
  HDG_CUDA(cudaGetLastError());
  s->ctx->launches++;
}
