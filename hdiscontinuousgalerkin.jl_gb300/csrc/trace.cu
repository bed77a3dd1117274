// Global trace system: deterministic gather of the condensed cell blocks into the trace matrix,
// and the Dirichlet treatment of apply!.
//
// The reference appends every cell's Ate as COO triplets and lets `sparse(I,J,V)` sort them and
// sum duplicates (src/assembler.jl:31-49).  Here the pattern is known from the topology: block
// row f (a face) holds nt x nt blocks for f itself and for the other faces of its one or two
// cells.  Each block has at most two sources (cell, local face pair): the diagonal block sums the
// blocks of the face's two cells, an off-diagonal block has exactly one.  The source map is built
// once per mesh, so assembly is an atomic-free gather; a sum of two terms does not depend on
// their order, so it reproduces the reference values exactly.
//
// Device layout (block-ELL, see hdg_internal.h): 5 slots per face, slot-major and
// row-contiguous, so every warp-wide load of the matrix in the CG is one contiguous segment.
#include <algorithm>

#include <numeric>

#include "hdg_device.cuh"

void build_block_structure(hdg_system* s) {
  const hdg_mesh* m = s->space->mesh;
  const int nf = m->nf;
  constexpr int S = hdg_system::SLOTS;
  s->h_browptr.assign(nf + 1, 0);
  s->h_bcol.clear();
  s->h_bsrc.clear();
  s->h_bcol.reserve((size_t)nf * S);
  s->h_bsrc.reserve((size_t)nf * S * 2);
  std::vector<int32_t> bcol5((size_t)S * nf), src5((size_t)S * nf * 2, -1);
  std::vector<int8_t> kdiag(nf, 0);
  int nb[8];
  for (int f = 0; f < nf; ++f) {
    const int c1 = m->faces[4 * f + 2], c2 = m->faces[4 * f + 3];
    int cnt = 0;
    nb[cnt++] = f;
    for (int c : {c1, c2}) {
      if (c < 0) continue;
      for (int l = 0; l < 3; ++l) {
        int g = m->cfaces[3 * c + l];
        if (g != f) nb[cnt++] = g;
      }
    }
    std::sort(nb, nb + cnt);
    cnt = (int)(std::unique(nb, nb + cnt) - nb);
    if (cnt > S) throw HdgError{HDG_ERR_ARG, "a face couples to more than 4 other faces (invalid triangle mesh)"};
    for (int k = 0; k < S; ++k) bcol5[(size_t)k * nf + f] = f;
    for (int k = 0; k < cnt; ++k) {
      const int g = nb[k];
      if (g == f) kdiag[f] = (int8_t)k;
      int src[2] = {-1, -1}, ns = 0;
      for (int c : {c1, c2}) {
        if (c < 0) continue;
        int lf = -1, lg = -1;
        for (int l = 0; l < 3; ++l) {
          if (m->cfaces[3 * c + l] == f) lf = l;
          if (m->cfaces[3 * c + l] == g) lg = l;
        }
        if (lf >= 0 && lg >= 0 && ns < 2) src[ns++] = c * 9 + lf * 3 + lg;
      }
      s->h_bcol.push_back(g);
      s->h_bsrc.push_back(src[0]);
      s->h_bsrc.push_back(src[1]);
      bcol5[(size_t)k * nf + f] = g;
      src5[((size_t)k * nf + f) * 2] = src[0];
      src5[((size_t)k * nf + f) * 2 + 1] = src[1];
    }
    s->h_browptr[f + 1] = (int32_t)s->h_bcol.size();
  }
  s->nblocks = (int64_t)s->h_bcol.size();
  s->nnz = s->nblocks * s->nt * s->nt;
  cudaStream_t st = s->ctx->stream;
  s->d_bcol5.upload(bcol5.data(), bcol5.size(), st);
  s->d_src5.upload(src5.data(), src5.size(), st);
  s->d_kdiag.upload(kdiag.data(), kdiag.size(), st);
  HDG_CUDA(cudaStreamSynchronize(st));
}

// Segments of the row-parallel kernels: every problem's trace rows are cut into ranges, one CUDA block each, so a block never
// spans two problems.
// A range has about 1024 rows (four per thread in the CG kernels).  Once the segments can fill the GPU, their number is
// rounded up to a multiple of the SM count (the extra segments go to the largest problems), so that every SM gets the
// same number of equal blocks.
// Far beyond one wave of resident blocks (4 to an SM in the FP64 iteration and all of multigrid, 6 in the FP32 one), a wave of
// longer ranges, as equal as the problems allow: a block spends 3 us on its reduction whatever its rows.  An iteration,
// us, segments of 1024 rows / 608 segments / 912: multigrid, 3.15 M rows of p = 3 473 / 436 / 460, 1.44 M of p = 2 332 / 318 /
// 333; FP64 Jacobi, 3.15 M rows 220 / 178 / 224; FP32 Jacobi 133 / 143 / 120.
SegCut cut_segments(const hdg_system* s, const char* on, bool fp32) {
  constexpr int64_t SEG_ROWS = 1024;
  const int np = s->nprob, sms = s->num_sm;
  auto rows_of = [&](int P) { return (int64_t)std::max(s->h_prob_row0[P + 1] - s->h_prob_row0[P], 1); };
  std::vector<int> of;
  int64_t longest = 1;
  for (int P = 0; P < np; ++P)
    if (!on || on[P]) {
      of.push_back(P);
      longest = std::max(longest, rows_of(P));
    }
  auto count = [&](int64_t len) {
    int64_t n = 0;
    for (int P : of) n += (rows_of(P) + len - 1) / len;
    return n;
  };
  int64_t len = SEG_ROWS, total = count(len);
  const int64_t wave = (int64_t)(fp32 ? 6 : 4) * sms;
  if (total > 8 * sms && (int64_t)of.size() <= wave) {  // the shortest ranges of which a wave holds all
    int64_t lo = len;
    for (len = longest; lo < len;) {
      const int64_t mid = (lo + len) / 2;
      if (count(mid) <= wave) len = mid;
      else lo = mid + 1;
    }
    total = count(len);
  }
  std::vector<int64_t> nseg(np, 0);
  for (int P : of) nseg[P] = (rows_of(P) + len - 1) / len;
  if (total >= sms) {
    int64_t extra = (sms - total % sms) % sms;
    std::vector<int> order(of);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return rows_of(x) > rows_of(y); });
    for (size_t k = 0; extra > 0; k = (k + 1) % order.size(), --extra) ++nseg[order[k]];
  }
  SegCut c;
  c.blk0.assign(np, 0);
  c.nblk.assign(np, 0);
  for (int P : of) {
    const int64_t a = s->h_prob_row0[P], e = s->h_prob_row0[P + 1], n = std::min(nseg[P], rows_of(P));
    const int64_t per = (rows_of(P) + n - 1) / n;
    c.blk0[P] = (int32_t)c.prob.size();
    c.nblk[P] = (int32_t)n;
    for (int64_t k = 0; k < n; ++k) {
      c.prob.push_back(P);
      c.row0.push_back((int32_t)std::min(e, a + k * per));
      c.row1.push_back((int32_t)std::min(e, a + (k + 1) * per));
    }
  }
  return c;
}

void put_segments(hdg_system* s, const SegCut& c, SegTable* t, cudaStream_t st) {
  const size_t n = c.prob.size(), np = (size_t)s->nprob;
  for (auto* b : {&t->d_prob, &t->d_row0, &t->d_row1}) b->alloc(s->seg_room);  // captured graphs hold the addresses
  for (auto* b : {&t->d_blk0, &t->d_nblk}) b->alloc(np);
  auto put = [&](DevBuf<int32_t>& to, const std::vector<int32_t>& v, size_t k) {
    HDG_CUDA(cudaMemcpyAsync(to.p, v.data(), k * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  };
  put(t->d_prob, c.prob, n);
  put(t->d_row0, c.row0, n);
  put(t->d_row1, c.row1, n);
  put(t->d_blk0, c.blk0, np);
  put(t->d_nblk, c.nblk, np);
  t->nseg = (int)n;
}

SegTable& segments_of(hdg_system* s, bool fp32) {
  if (fp32 && !s->seg32_known) {
    s->seg32_known = true;
    SegCut c = cut_segments(s, nullptr, true);
    if (c.prob.size() != s->seg.full.prob.size()) {
      put_segments(s, c, &s->seg32, s->ctx->stream);
      HDG_CUDA(cudaStreamSynchronize(s->ctx->stream));  // the solve's stream may be another
      s->seg32.full = std::move(c);
    }
  }
  return fp32 && s->seg32.nseg > 0 ? s->seg32 : s->seg;
}

void build_segments(hdg_system* s) {
  const hdg_mesh* m = s->space->mesh;
  s->nprob = m->nprob;
  HDG_CUDA(cudaDeviceGetAttribute(&s->num_sm, cudaDevAttrMultiProcessorCount, s->ctx->device));
  s->h_prob_row0.assign(s->nprob + 1, 0);
  std::vector<int32_t> rowp((size_t)s->ndofs);
  size_t all = 0;
  for (int P = 0; P < s->nprob; ++P) {
    s->h_prob_row0[P] = m->prob_face0[P] * s->nt;
    s->h_prob_row0[P + 1] = m->prob_face0[P + 1] * s->nt;
    all += std::max(s->h_prob_row0[P + 1] - s->h_prob_row0[P], 1) / 1024 + 1;
    for (int r = s->h_prob_row0[P]; r < s->h_prob_row0[P + 1]; ++r) rowp[r] = P;
  }
  // segments of 1024 rows and the extra ones; beyond 8 to an SM only where a wave is too few for the problems
  s->seg_room = all + s->num_sm;
  if (s->nprob <= 4 * s->num_sm) s->seg_room = std::min(s->seg_room, (size_t)9 * s->num_sm);
  SegCut c = cut_segments(s, nullptr, false);
  put_segments(s, c, &s->seg, s->ctx->stream);
  s->seg.full = std::move(c);
  cudaStream_t st = s->ctx->stream;
  s->d_row_prob.upload(rowp.data(), rowp.size(), st);
  s->ensure_reduction_buffers();
  HDG_CUDA(cudaStreamSynchronize(st));
}

namespace {
constexpr int S5 = hdg_system::SLOTS;

// Assembly of the trace system from the condensed blocks, GF faces per CTA:
//   val[(k nt + j) ndofs + r] = sum over sources of Ate_c[lf nt + i, lg nt + j],  r = f nt + i
//   b[r] = sum over the face's cells of bte_c[lf nt + i]        (assemble!(K, gdof, Ate) and (b, gdof, bte))
// The CTA first copies, for each of its faces and each of the face's two cells, the cell's nt rows of
// [Ate | bte] that belong to the face (one contiguous run of nt (m+1) doubles) into shared memory,
// then writes the faces' 5 nt x nt slot blocks slot-major, so that both the reads and the writes
// are contiguous.  The sources of a slot are added in the order src5 lists them (first the face's
// first cell), the right-hand side's in the face's cell order.  Shared rows are padded to an odd
// number of doubles so that the threads of a half-warp (consecutive rows of consecutive faces)
// fall on different banks.
template <int NT> struct GatherTile {
  static constexpr int M = 3 * NT, MS = M + 1;
  static constexpr int MSP = MS | 1;                             // padded row
  static constexpr int RBP = (NT * MSP) | 1;                     // padded row block (one face, one cell)
  static constexpr int GF = 32;                                  // faces per CTA
  static constexpr size_t SMEM = sizeof(double) * (size_t)GF * 2 * RBP;
};

template <int NT>
__global__ void __launch_bounds__(256) k_gather_faces(const int nf, const int32_t* __restrict__ fcell,
                                                      const int8_t* __restrict__ flf,
                                                      const int32_t* __restrict__ src5,
                                                      const double* __restrict__ AB, double* __restrict__ val,
                                                      double* __restrict__ b) {
  using T = GatherTile<NT>;
  constexpr int M = T::M, MS = T::MS, MSP = T::MSP, RBP = T::RBP, GF = T::GF, RB = NT * MS;
  extern __shared__ double sm[];
  const int f0 = blockIdx.x * GF;
  const int nfb = min(GF, nf - f0);
  for (int t = threadIdx.x; t < nfb * 2 * RB; t += blockDim.x) {
    const int fq = t / RB, e = t - fq * RB;                  // fq = 2 (face in tile) + side
    const int c = fcell[2 * f0 + fq];
    const int i = e / MS, col = e - i * MS;
    sm[fq * RBP + i * MSP + col] = c >= 0 ? AB[(int64_t)c * M * MS + (int64_t)flf[2 * f0 + fq] * RB + e] : 0.0;
  }
  __syncthreads();
  const int64_t ndofs = (int64_t)nf * NT;
  const int nr = nfb * NT;                                       // rows of the tile
  for (int t = threadIdx.x; t < S5 * NT * nr; t += blockDim.x) {
    const int sl = t / nr, r = t - sl * nr;
    const int fl = r / NT, i = r - fl * NT, k = sl / NT, j = sl - k * NT;
    const int f = f0 + fl;
    const int2 sp = *reinterpret_cast<const int2*>(src5 + ((int64_t)k * nf + f) * 2);
    const int c1 = fcell[2 * f];
    double v = 0.0;
    if (sp.x >= 0) v += sm[(2 * fl + (sp.x / 9 == c1 ? 0 : 1)) * RBP + i * MSP + (sp.x % 3) * NT + j];
    if (sp.y >= 0) v += sm[(2 * fl + (sp.y / 9 == c1 ? 0 : 1)) * RBP + i * MSP + (sp.y % 3) * NT + j];
    val[(int64_t)sl * ndofs + (int64_t)f0 * NT + r] = v;
  }
  for (int r = threadIdx.x; r < nr; r += blockDim.x) {
    const int fl = r / NT, i = r - fl * NT;
    double v = 0.0;
    v += sm[(2 * fl) * RBP + i * MSP + M];
    if (fcell[2 * (f0 + fl) + 1] >= 0) v += sm[(2 * fl + 1) * RBP + i * MSP + M];
    b[(int64_t)f0 * NT + r] = v;
  }
}

// meandiag(K) = mean |K_ii| of each problem (src/boundary.jl:169-175), a deterministic
// per-problem reduction over the segments.
template <int NT>
__global__ void k_meandiag(SegArgs g, const int32_t* __restrict__ prob_row0, const int nf,
                           const int8_t* __restrict__ kdiag, const double* __restrict__ val, double* __restrict__ mdiag) {
  const int P = g.seg_prob[blockIdx.x];
  const int ndofs = nf * NT;
  double acc = 0.0;
  for (int r = g.seg_row0[blockIdx.x] + threadIdx.x; r < g.seg_row1[blockIdx.x]; r += blockDim.x) {
    const int f = r / NT, i = r - f * NT;
    acc += fabs(val[(int64_t)(kdiag[f] * NT + i) * ndofs + r]);
  }
  double s0;
  if (seg_finish1<256>(g, P, 3, acc, &s0) && threadIdx.x == 0)
    mdiag[P] = s0 / (double)(prob_row0[P + 1] - prob_row0[P]);
}

// b -= sum_d v_d K[:, d] over prescribed dofs with v_d != 0 (src/boundary.jl:128-137); gv holds
// v at prescribed dofs and 0 elsewhere, so this is one sparse product with gv.
template <int NT>
__global__ void k_lift(const int nf, const int32_t* __restrict__ bcol5, const double* __restrict__ val,
                       const double* __restrict__ gv, double* __restrict__ b) {
  const int ndofs = nf * NT;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= ndofs) return;
  const int f = r / NT;
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < S5; ++k) {
    const int g = bcol5[k * nf + f];
#pragma unroll
    for (int j = 0; j < NT; ++j) s += val[(int64_t)(k * NT + j) * ndofs + r] * gv[g * NT + j];
  }
  b[r] -= s;
}

// Rows and columns of prescribed dofs zeroed, K[d,d] = m, b[d] = v m (src/boundary.jl:138-157).
// The result is stored in "solver form": free rows negated, so that the matrix the CG sees is
// symmetric positive definite (the condensed HDG trace operator is negative definite on the free
// dofs).  hdg_system_get_csc undoes the sign when exporting.
template <int NT>
__global__ void k_apply(const int nf, const int32_t* __restrict__ bcol5, const int8_t* __restrict__ kdiag,
                        const uint8_t* __restrict__ pres, const double* __restrict__ gv, const double* __restrict__ md,
                        const int32_t* __restrict__ row_prob, double* __restrict__ val, double* __restrict__ b) {
  const int ndofs = nf * NT;
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= ndofs) return;
  const int f = r / NT, i = r - f * NT, kd = kdiag[f];
  const double m = md[row_prob[r]];
  const bool pr = pres[r];
#pragma unroll
  for (int k = 0; k < S5; ++k) {
    const int g = bcol5[k * nf + f];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      double& v = val[(int64_t)(k * NT + j) * ndofs + r];
      if (pr || pres[g * NT + j]) v = (k == kd && j == i) ? m : 0.0;
      else v = -v;
    }
  }
  b[r] = pr ? gv[r] * m : -b[r];
}

// prescribed dofs -> per-dof flag and value
__global__ void k_scatter_dirichlet(const int n, const int32_t* __restrict__ dofs, const double* __restrict__ vals,
                                    uint8_t* __restrict__ pres, double* __restrict__ gv) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  pres[dofs[k]] = 1;
  gv[dofs[k]] = vals[k];
}

// The columns of faces g0 .. g1 - 1 as CSC, in the signs the reference holds them: column g NT + j holds K[f NT + i, g NT + j] of the
// block rows f that couple to g (the pattern is symmetric, so these are g's own neighbours, ascending).  One warp per
// face: the lanes find the slot of g in each neighbour's row, then write the face's entries in their order, consecutive
// lanes consecutive addresses; e0 = the first entry of g0.  What bounds an export is the caller's memory: for the 2.2 million
// entries of 2 x 96^2 cells of p = 3 a host loop over the downloaded slots took 4.7 ms; now the pages of fresh arrays
// take 1.1 ms and this kernel and the copies 0.35.
template <int NT>
__global__ void k_export_csc(const int g0, const int g1, const int nf, const int64_t base, const int32_t* __restrict__ browptr,
                             const int32_t* __restrict__ bcol5, const double* __restrict__ val,
                             const double* __restrict__ b, const uint8_t* __restrict__ pres, int64_t* __restrict__ colptr,
                             int64_t* __restrict__ rowval, double* __restrict__ nzval, double* __restrict__ rhs) {
  const int g = g0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (g >= g1) return;
  const int64_t ndofs = (int64_t)nf * NT;
  const int deg = browptr[g + 1] - browptr[g];
  const int64_t first = (int64_t)NT * NT * browptr[g], e0 = (int64_t)NT * NT * browptr[g0];
  int fk = 0, kp = -1;
  if (lane < deg) {
    fk = bcol5[lane * nf + g];
    const int df = browptr[fk + 1] - browptr[fk];
    for (int q = df - 1; q >= 0; --q)
      if (bcol5[q * nf + fk] == g) kp = q;
  }
  for (int t0 = 0; t0 < NT * NT * deg; t0 += 32) {
    const int t = t0 + lane, j = t / (NT * deg), r = t - j * NT * deg, k = r / NT, i = r - k * NT;
    const int f = __shfl_sync(0xffffffffu, fk, k & 31), q = __shfl_sync(0xffffffffu, kp, k & 31);
    if (t >= NT * NT * deg) break;
    const int64_t row = (int64_t)f * NT + i;
    if (rowval) rowval[first - e0 + t] = row + base;
    if (nzval) {
      const double v = q >= 0 ? val[(int64_t)(q * NT + j) * ndofs + row] : 0.0;
      nzval[first - e0 + t] = pres && !pres[row] ? -v : v;
    }
  }
  if (lane < NT) {
    const int64_t row = (int64_t)g * NT + lane, at = (int64_t)(g - g0) * NT + lane;
    if (colptr) colptr[at] = first + (int64_t)(lane + 1) * NT * deg + base;  // the end of column row
    if (rhs) rhs[at] = pres && !pres[row] ? -b[row] : b[row];
  }
}

template <int NT> void gather_t(hdg_system* s, cudaStream_t st) {
  using T = GatherTile<NT>;
  hdg_mesh* m = s->space->mesh;
  if (m->nf <= 0) return;
  const unsigned blocks = (unsigned)((m->nf + T::GF - 1) / T::GF);
  k_gather_faces<NT><<<blocks, 256, T::SMEM, st>>>(m->nf, m->d_fcell.p, m->d_flf.p, s->d_src5.p, s->d_AB.p,
                                                    s->d_val.p, s->d_b.p);
  HDG_CUDA(cudaGetLastError());
  s->ctx->launches += 1;
}

// Scatter of the prescribed dofs and values into per-row flags and values (d_pres, d_gv): the
// part of apply! that depends only on the Dirichlet data, so it survives reassembly.
void dirichlet_scatter(hdg_system* s, const std::vector<int32_t>& dofs0, const std::vector<double>& vals,
                       cudaStream_t st) {
  const int nrow = s->ndofs;
  bool lift = false;
  for (size_t k = 0; k < dofs0.size(); ++k)
    if (vals[k] != 0.0) lift = true;
  s->ensure_reduction_buffers();
  s->d_pres.alloc(nrow);
  s->d_gv.alloc(nrow);
  HDG_CUDA(cudaMemsetAsync(s->d_pres.p, 0, nrow, st));
  HDG_CUDA(cudaMemsetAsync(s->d_gv.p, 0, nrow * sizeof(double), st));
  const int nd = (int)dofs0.size();
  if (nd > 0) {
    s->d_dofs.upload(dofs0.data(), nd, st);
    s->d_dvals.upload(vals.data(), nd, st);
    k_scatter_dirichlet<<<(nd + 255) / 256, 256, 0, st>>>(nd, s->d_dofs.p, s->d_dvals.p, s->d_pres.p, s->d_gv.p);
    HDG_CUDA(cudaGetLastError());
    s->ctx->launches++;
  }
  s->d_mdiag.alloc(s->nprob);
  s->d_prob_row0_dev();
  s->dir_lift = lift;
  s->dir_ready = true;
}

// apply! on the assembled system from the scattered Dirichlet data: per-problem mean |diag|,
// lifting of the prescribed values into b, and the symmetric row/column elimination.
template <int NT> void apply_t(hdg_system* s, cudaStream_t st) {
  hdg_mesh* m = s->space->mesh;
  const int nrow = m->nf * NT;
  const SegTable& t = s->seg;
  const SegArgs g{t.d_prob.p, t.d_row0.p, t.d_row1.p, t.d_blk0.p, t.d_nblk.p, s->d_part.p, s->d_cnt.p};
  k_meandiag<NT><<<t.nseg, 256, 0, st>>>(g, s->d_prob_row0.p, m->nf, s->d_kdiag.p, s->d_val.p, s->d_mdiag.p);
  HDG_CUDA(cudaGetLastError());
  if (s->dir_lift) {
    k_lift<NT><<<(nrow + 255) / 256, 256, 0, st>>>(m->nf, s->d_bcol5.p, s->d_val.p, s->d_gv.p, s->d_b.p);
    HDG_CUDA(cudaGetLastError());
    s->ctx->launches++;
  }
  k_apply<NT><<<(nrow + 255) / 256, 256, 0, st>>>(m->nf, s->d_bcol5.p, s->d_kdiag.p, s->d_pres.p, s->d_gv.p,
                                                  s->d_mdiag.p, s->d_row_prob.p, s->d_val.p, s->d_b.p);
  HDG_CUDA(cudaGetLastError());
  s->ctx->launches += 2;
}

template <int NT>
void export_csc_t(const hdg_system* s, int base, int64_t* colptr, int64_t* rowval, double* nzval, double* rhs,
                  cudaStream_t st) {
  const int nf = s->nf, per_face = NT * NT * hdg_system::SLOTS;
  // staged in pieces of at most 2 million entries, 32 MB on the device whatever the system
  const int faces = std::min(nf, std::max(1, (1 << 21) / per_face));
  DevBuf<int32_t> browptr;
  DevBuf<int64_t> cp, rv;
  DevBuf<double> nz, rh;
  browptr.upload(s->h_browptr.data(), s->h_browptr.size(), st);
  if (colptr) cp.alloc((size_t)faces * NT);
  if (rowval) rv.alloc((size_t)faces * per_face);
  if (nzval) nz.alloc((size_t)faces * per_face);
  if (rhs) rh.alloc((size_t)faces * NT);
  for (int g0 = 0; g0 < nf; g0 += faces) {
    const int g1 = std::min(nf, g0 + faces);
    k_export_csc<NT><<<(unsigned)((g1 - g0 + 7) / 8), 256, 0, st>>>(g0, g1, nf, base, browptr.p, s->d_bcol5.p, s->d_val.p,
                                                                    s->d_b.p, s->applied ? s->d_pres.p : nullptr, cp.p, rv.p,
                                                                    nz.p, rh.p);
    HDG_CUDA(cudaGetLastError());
    s->ctx->launches++;
    const size_t e0 = (size_t)NT * NT * s->h_browptr[g0], ne = (size_t)NT * NT * s->h_browptr[g1] - e0;
    const size_t r0 = (size_t)g0 * NT, nr = (size_t)(g1 - g0) * NT;
    if (colptr) populate_pages(colptr + 1 + r0, nr * sizeof(int64_t));
    if (rowval) populate_pages(rowval + e0, ne * sizeof(int64_t));
    if (nzval) populate_pages(nzval + e0, ne * sizeof(double));
    if (rhs) populate_pages(rhs + r0, nr * sizeof(double));
    if (colptr) cp.download(colptr + 1 + r0, nr, st);
    if (rowval) rv.download(rowval + e0, ne, st);
    if (nzval) nz.download(nzval + e0, ne, st);
    if (rhs) rh.download(rhs + r0, nr, st);
  }
  HDG_CUDA(cudaStreamSynchronize(st));
}

}  // namespace

void run_export_csc(const hdg_system* s, int base, int64_t* colptr, int64_t* rowval, double* nzval, double* rhs,
                    cudaStream_t st) {
  if (colptr) colptr[0] = base;
  switch (s->nt) {
    case 2: return export_csc_t<2>(s, base, colptr, rowval, nzval, rhs, st);
    case 3: return export_csc_t<3>(s, base, colptr, rowval, nzval, rhs, st);
    case 4: return export_csc_t<4>(s, base, colptr, rowval, nzval, rhs, st);
    case 5: return export_csc_t<5>(s, base, colptr, rowval, nzval, rhs, st);
    default: throw HdgError{HDG_ERR_ARG, "degree not supported"};
  }
}

void launch_gather(hdg_system* s, cudaStream_t st) {
  switch (s->nt) {
    case 2: gather_t<2>(s, st); break;
    case 3: gather_t<3>(s, st); break;
    case 4: gather_t<4>(s, st); break;
    case 5: gather_t<5>(s, st); break;
    default: throw HdgError{HDG_ERR_ARG, "degree not supported"};
  }
}

void launch_dirichlet_scatter(hdg_system* s, const std::vector<int32_t>& dofs0, const std::vector<double>& vals,
                              cudaStream_t st) {
  dirichlet_scatter(s, dofs0, vals, st);
}

void launch_dirichlet_apply(hdg_system* s, cudaStream_t st) {
  if (!s->dir_ready) throw HdgError{HDG_ERR_ARG, "no Dirichlet set was given to this system"};
  switch (s->nt) {
    case 2: apply_t<2>(s, st); break;
    case 3: apply_t<3>(s, st); break;
    case 4: apply_t<4>(s, st); break;
    case 5: apply_t<5>(s, st); break;
    default: throw HdgError{HDG_ERR_ARG, "degree not supported"};
  }
}

void launch_apply_dirichlet(hdg_system* s, const std::vector<int32_t>& dofs0, const std::vector<double>& vals,
                            cudaStream_t st) {
  launch_dirichlet_scatter(s, dofs0, vals, st);
  launch_dirichlet_apply(s, st);
}
