// C ABI of libhdg (include/hdg.h): argument checking, object lifetimes, error reporting.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cerrno>
#include <cmath>
#include <cstring>
#include <functional>

#include "hdg_internal.h"

namespace {

thread_local std::string g_err;  // for failures before a context exists

int guard(hdg_ctx* ctx, const std::function<int()>& fn) {
  try {
    int rc = fn();
    return rc;
  } catch (const HdgError& e) {
    if (ctx) ctx->err = e.msg;
    g_err = e.msg;
    return e.code;
  } catch (const std::bad_alloc&) {
    if (ctx) ctx->err = "host allocation failed";
    g_err = "host allocation failed";
    return HDG_ERR_OOM;
  } catch (const std::exception& e) {
    if (ctx) ctx->err = e.what();
    g_err = e.what();
    return HDG_ERR_ARG;
  }
}

int fail(hdg_ctx* ctx, int code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  g_err = msg;
  return code;
}

void set_device(hdg_ctx* ctx) {
  HDG_CUDA(cudaSetDevice(ctx->device));
  g_alloc_stream = ctx->stream;
}

}  // namespace

thread_local cudaStream_t g_alloc_stream = nullptr;
thread_local cudaStream_t g_use_stream = nullptr;
thread_local bool g_tuning_allowed = true;

void order_streams(cudaStream_t before, cudaStream_t after) {
  cudaEvent_t e;
  HDG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  HDG_CUDA(cudaEventRecord(e, before));
  HDG_CUDA(cudaStreamWaitEvent(after, e, 0));
  HDG_CUDA(cudaEventDestroy(e));
}

hdg_system::~hdg_system() {
  if (cg) destroy_cg(cg);
  if (amg) destroy_amg(amg);
  for (auto* e : ev_cg_a) delete e;
  for (auto* e : ev_cg_b) delete e;
  for (auto* e : ev_res) delete e;
  for (auto* e : ev_cheb0) delete e;
  for (auto* e : ev_l1) delete e;
}

extern "C" {

int hdg_ctx_create(int device, hdg_ctx** out) {
  if (!out) return HDG_ERR_ARG;
  return guard(nullptr, [&]() -> int {
    int n = 0;
    HDG_CUDA(cudaGetDeviceCount(&n));
    if (device < 0 || device >= n) return fail(nullptr, HDG_ERR_ARG, "no such CUDA device");
    hdg_ctx* c = new hdg_ctx();
    c->device = device;
    HDG_CUDA(cudaSetDevice(device));
    HDG_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    c->own_stream = true;
    // keep freed blocks in this process's pool instead of returning them to the driver
    cudaMemPool_t pool;
    HDG_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    uint64_t keep = UINT64_MAX;
    HDG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    *out = c;
    return HDG_OK;
  });
}

int hdg_ctx_destroy(hdg_ctx* ctx) {
  if (!ctx) return HDG_OK;
  cudaSetDevice(ctx->device);
  if (ctx->own_stream && ctx->stream) {
    cudaStreamSynchronize(ctx->stream);
    cudaStreamDestroy(ctx->stream);
  }
  delete ctx;
  return HDG_OK;
}

const char* hdg_last_error(const hdg_ctx* ctx) { return ctx ? ctx->err.c_str() : g_err.c_str(); }

int hdg_ctx_set_stream(hdg_ctx* ctx, void* stream) {
  if (!ctx) return HDG_ERR_ARG;
  return guard(ctx, [&]() -> int {
    set_device(ctx);
    if (ctx->own_stream && ctx->stream) {
      HDG_CUDA(cudaStreamSynchronize(ctx->stream));
      HDG_CUDA(cudaStreamDestroy(ctx->stream));
    }
    if (stream) {
      ctx->stream = (cudaStream_t)stream;
      ctx->own_stream = false;
    } else {
      HDG_CUDA(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
      ctx->own_stream = true;
    }
    return HDG_OK;
  });
}

int64_t hdg_ctx_launch_count(const hdg_ctx* ctx) { return ctx ? ctx->launches : 0; }

int hdg_ctx_set_profiling(hdg_ctx* ctx, int on) {
  if (!ctx) return HDG_ERR_ARG;
  ctx->profiling = on != 0;
  return HDG_OK;
}

// ---------------------------------------------------------------- mesh
// A NULL context builds a host-only mesh (topology queries only; no space can be built on it).
int hdg_mesh_rectangle(hdg_ctx* ctx, int nx, int ny, const double LL[2], const double UR[2], hdg_mesh** out) {
  if (!out || nx < 1 || ny < 1 || !LL || !UR) return fail(ctx, HDG_ERR_ARG, "hdg_mesh_rectangle: bad arguments");
  if ((double)nx * ny * 3.0 + nx + ny > 2.0e9) return fail(ctx, HDG_ERR_ARG, "mesh too large for 32-bit face ids");
  return guard(ctx, [&]() -> int {
    if (ctx) set_device(ctx);
    hdg_mesh* m = new hdg_mesh();
    m->ctx = ctx;
    try {
      mesh_build_rectangle(m, nx, ny, LL, UR);
      if (ctx) m->upload();
    } catch (...) {
      delete m;
      throw;
    }
    *out = m;
    return HDG_OK;
  });
}

int hdg_mesh_from_cells(hdg_ctx* ctx, int nnodes, const double* xy, int ncells, const int32_t* cell_nodes, int nedges,
                        const int32_t* edges, hdg_mesh** out) {
  if (!out || nnodes < 3 || ncells < 1 || !xy || !cell_nodes || (nedges > 0 && !edges))
    return fail(ctx, HDG_ERR_ARG, "hdg_mesh_from_cells: bad arguments");
  return guard(ctx, [&]() -> int {
    if (ctx) set_device(ctx);
    hdg_mesh* m = new hdg_mesh();
    m->ctx = ctx;
    int rc = mesh_build_from_cells(m, nnodes, xy, ncells, cell_nodes, nedges, edges);
    if (rc != HDG_OK) {
      delete m;
      return fail(ctx, rc, "hdg_mesh_from_cells: node id out of range");
    }
    try {
      if (ctx) m->upload();
    } catch (...) {
      delete m;
      throw;
    }
    *out = m;
    return HDG_OK;
  });
}

int hdg_mesh_set_coordinates(hdg_mesh* m, const double* xy) {
  if (!m || !xy) return HDG_ERR_ARG;
  return guard(m->ctx, [&]() -> int {
    std::memcpy(m->xy.data(), xy, m->xy.size() * sizeof(double));
    if (!m->ctx) return HDG_OK;
    set_device(m->ctx);
    m->upload_coordinates();
    return HDG_OK;
  });
}

int hdg_mesh_jitter(hdg_mesh* m, double a, uint64_t seed) {
  if (!m || !m->structured || !(a >= 0.0) || a >= 0.35)
    return fail(m ? m->ctx : nullptr, HDG_ERR_ARG, "hdg_mesh_jitter: needs a rectangle mesh and 0 <= a < 0.35");
  return guard(m->ctx, [&]() -> int {
    const double hx = (m->UR[0] - m->LL[0]) / m->nx, hy = (m->UR[1] - m->LL[1]) / m->ny;
    uint64_t st = seed ^ 0x9E3779B97F4A7C15ull;
    auto next = [&]() {  // splitmix64 -> uniform in [-1, 1)
      uint64_t z = (st += 0x9E3779B97F4A7C15ull);
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      z ^= z >> 31;
      return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    const int NX = m->nx + 1;
    for (int j = 1; j < m->ny; ++j)
      for (int i = 1; i < m->nx; ++i) {
        double* p = &m->xy[2 * ((size_t)j * NX + i)];
        p[0] += a * hx * next();
        p[1] += a * hy * next();
      }
    if (!m->ctx) return HDG_OK;
    set_device(m->ctx);
    m->upload_coordinates();
    HDG_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return HDG_OK;
  });
}

int hdg_mesh_sizes(const hdg_mesh* m, int* nn, int* nc, int* nf) {
  if (!m) return HDG_ERR_ARG;
  if (nn) *nn = m->nn;
  if (nc) *nc = m->nc;
  if (nf) *nf = m->nf;
  return HDG_OK;
}

int hdg_mesh_get_topology(const hdg_mesh* m, double* xy, int32_t* cell_nodes, int32_t* cell_faces, int32_t* faces) {
  if (!m) return HDG_ERR_ARG;
  if (xy) std::memcpy(xy, m->xy.data(), m->xy.size() * sizeof(double));
  if (cell_nodes)
    for (size_t i = 0; i < m->cells.size(); ++i) cell_nodes[i] = m->cells[i] + 1;
  if (cell_faces)
    for (size_t i = 0; i < m->cfaces.size(); ++i) cell_faces[i] = m->cfaces[i] + 1;
  if (faces)
    for (size_t i = 0; i < m->faces.size(); ++i) faces[i] = m->faces[i] + 1;  // c2 = -1 -> 0
  return HDG_OK;
}

int hdg_mesh_faceset(const hdg_mesh* m, const char* name, int32_t* out, int* count) {
  if (!m || !name || !count) return HDG_ERR_ARG;
  auto it = m->facesets.find(name);
  if (it == m->facesets.end()) return fail(m->ctx, HDG_ERR_UNKNOWN_SET, std::string("no face set ") + name);
  *count = (int)it->second.size();
  if (out)
    for (size_t i = 0; i < it->second.size(); ++i) out[i] = it->second[i] + 1;
  return HDG_OK;
}

int hdg_mesh_destroy(hdg_mesh* m) {
  if (m) {
    if (m->ctx) {
      cudaSetDevice(m->ctx->device);
      cudaStreamSynchronize(m->ctx->stream);
    }
    delete m;
  }
  return HDG_OK;
}

// ---------------------------------------------------------------- spaces
int hdg_space_create(hdg_mesh* mesh, int p, int qd, hdg_space** out) {
  if (!mesh || !out) return HDG_ERR_ARG;
  hdg_ctx* ctx = mesh->ctx;
  if (!ctx) return fail(nullptr, HDG_ERR_ARG, "the mesh was built without a device context");
  if (p < 1 || p > HDG_MAX_P) return fail(ctx, HDG_ERR_ARG, "degree must be 1..4");
  if (qd <= 0) qd = p + 1;
  return guard(ctx, [&]() -> int {
    set_device(ctx);
    hdg_space* s = new hdg_space();
    s->mesh = mesh;
    if (!build_ref_tables(p, qd, &s->t)) {
      delete s;
      return fail(ctx, HDG_ERR_BAD_ORDER, "Quadrature rule of order " + std::to_string(qd) + " not available");
    }
    s->d_ref.upload(s->t.packed.data(), s->t.packed.size(), ctx->stream);
    HDG_CUDA(cudaStreamSynchronize(ctx->stream));
    *out = s;
    return HDG_OK;
  });
}

int hdg_space_info(const hdg_space* s, int* nw, int* nv, int* nt, int* nq, int* nfq) {
  if (!s) return HDG_ERR_ARG;
  if (nw) *nw = s->t.nw;
  if (nv) *nv = 2 * s->t.nw;
  if (nt) *nt = s->t.nt;
  if (nq) *nq = s->t.nq;
  if (nfq) *nfq = s->t.nfq;
  return HDG_OK;
}

int hdg_space_tables(const hdg_space* s, double* pts, double* w, double* N, double* dN, double* fpts, double* fw,
                     double* E, double* T) {
  if (!s) return HDG_ERR_ARG;
  const RefTables& t = s->t;
  if (pts)
    for (int q = 0; q < t.nq; ++q) { pts[2 * q] = t.qx[q]; pts[2 * q + 1] = t.qy[q]; }
  if (w) std::memcpy(w, t.qw.data(), t.nq * sizeof(double));
  if (N) std::memcpy(N, t.N.data(), t.N.size() * sizeof(double));
  if (dN) std::memcpy(dN, t.dN.data(), t.dN.size() * sizeof(double));
  if (fpts) std::memcpy(fpts, t.fx.data(), t.nfq * sizeof(double));
  if (fw) std::memcpy(fw, t.fw.data(), t.nfq * sizeof(double));
  if (E) std::memcpy(E, t.E.data(), t.E.size() * sizeof(double));
  if (T) std::memcpy(T, t.T.data(), t.T.size() * sizeof(double));
  return HDG_OK;
}

int hdg_space_cell_geometry(const hdg_space* s, int cell, double* detJ, double* Jinv, double* detJf, double* nrm) {
  if (!s || cell < 1 || cell > s->mesh->nc) return fail(s ? s->mesh->ctx : nullptr, HDG_ERR_ARG, "bad cell");
  const hdg_mesh* m = s->mesh;
  const int c = cell - 1;
  const double* X[3] = {&m->xy[2 * m->cells[3 * c]], &m->xy[2 * m->cells[3 * c + 1]], &m->xy[2 * m->cells[3 * c + 2]]};
  const double J00 = X[1][0] - X[0][0], J01 = X[2][0] - X[0][0], J10 = X[1][1] - X[0][1], J11 = X[2][1] - X[0][1];
  const double d = J00 * J11 - J01 * J10;
  if (!(d > 0.0)) return fail(m->ctx, HDG_ERR_NEG_DETJ, "det(J) is not positive: det(J) = " + std::to_string(d));
  if (detJ) *detJ = d;
  if (Jinv) { Jinv[0] = J11 / d; Jinv[1] = -J01 / d; Jinv[2] = -J10 / d; Jinv[3] = J00 / d; }
  const double wn[3][2] = {{-(J10 - J11), J00 - J01}, {-J11, J01}, {J10, -J00}};
  for (int f = 0; f < 3; ++f) {
    const double l = std::sqrt(wn[f][0] * wn[f][0] + wn[f][1] * wn[f][1]);
    if (detJf) detJf[f] = l;
    if (nrm) { nrm[2 * f] = wn[f][0] / l; nrm[2 * f + 1] = wn[f][1] / l; }
  }
  return HDG_OK;
}

int hdg_space_destroy(hdg_space* s) {
  delete s;
  return HDG_OK;
}

// ---------------------------------------------------------------- fields in fixed point
// hdg_device.cuh: eval_part.  A problem's coordinates are below 2^e in magnitude, its fixed-point numbers are X = x 2^s.
// FP64 holds a coordinate to 2^-53 of its own magnitude, the fixed point every one to 2^-s; a field takes the fixed form
// only where the latter costs it nothing against the former, and no other problem of the system has a say in it.

static int coordinate_exponent(double xy_max) {  // smallest e with xy_max < 2^e
  int e;
  std::frexp(xy_max, &e);
  return e;
}

// A bump that adds nothing anywhere below 2^e: of amplitude 0, or so far off that its exponential is 0 in FP64
// (exp(-x) from x = 745.2 on, 38.7 widths).
static bool bump_is_off(const double* b, int e) {
  const double edge = std::ldexp(1.0, e), dx = std::max(std::fabs(b[0]) - edge, 0.0), dy = std::max(std::fabs(b[1]) - edge, 0.0);
  return b[3] == 0.0 || std::hypot(dx, dy) > 38.7 * std::fabs(b[2]);
}
static bool bumps_finite(const std::vector<double>& p) {
  return std::all_of(p.begin() + 1, p.begin() + 1 + 4 * (int)p[0], [](double v) { return std::isfinite(v); });
}

// The exponent of one problem's fixed point: above its coordinates and the centres of the bumps that matter to it.
static int fixed_exponent(int e, const FieldSpec& f) {
  if (f.kind != HDG_FIELD_BUMPS || !bumps_finite(f.prm)) return e;
  int top = e;
  for (int k = 0; k < (int)f.prm[0]; ++k) {
    const double* b = &f.prm[1 + 4 * k];
    if (!bump_is_off(b, e)) top = std::max(top, coordinate_exponent(std::max(std::fabs(b[0]), std::fabs(b[1]))));
  }
  return top;
}

// Rewrites the parameters of one field at prm (its FieldSpec's, in place) for coordinates X = x 2^s, |x| < 2^e, and
// returns the fixed-point kind, or leaves them (a Gaussian's width prepared as in fprep) and returns the plain one where
// a value does not fit the form or the form would lose digits to FP64.
static int prepare_fixed(const FieldSpec& f, int s, int e, bool usable, double* prm) {
  auto word = [](uint64_t v) {
    double d;
    std::memcpy(&d, &v, 8);
    return d;
  };
  auto ceil_log2 = [](double v) {  // smallest e with v <= 2^e
    int e;
    const double m = std::frexp(v, &e);
    return m == 0.5 ? e - 1 : e;
  };
  const std::vector<double>& p = f.prm;
  const int K = (f.kind == HDG_FIELD_BUMPS || f.kind == HDG_FIELD_FOURIER || f.kind == HDG_FIELD_EXP_FOURIER) ? (int)p[0] : 0;
  if (f.kind == HDG_FIELD_BUMPS) {
    bool fits = usable && bumps_finite(p);
    std::vector<uint64_t> w;
    w.reserve(4 * (size_t)K);
    for (int k = 0; k < K && fits; ++k) {
      const double* b = &p[1 + 4 * k];
      if (b[2] != 0.0 && bump_is_off(b, e)) continue;
      // A bump is wide against the grid, or lies where FP64's own spacing of the coordinates is no finer: 2^-s at most
      // 2^-54 of the larger.
      const double size = std::max(std::max(std::fabs(b[0]), std::fabs(b[1])), std::fabs(b[2]));
      fits = b[2] != 0.0 && size >= std::ldexp(1.0, 54 - s);
      if (!fits) break;
      // |dx| 2^s scaled to r sqrt(log2 e / 2) / sigma in units of 2^-59: a factor below 2^64 and a shift
      const long double c = 0.84932180028801904272L / std::fabs((long double)b[2]);
      int ec;
      const long double m = std::frexp(c, &ec);  // c = m 2^ec, m in [1/2, 1)
      const int up = ec + 59 - s;                // G = |dx| m 2^up
      const int sh = std::max(0, up);
      fits = sh <= 62 && up > -200;
      if (!fits) break;
      const long double q = std::ldexp(m, 64 + up - sh);  // at most 2^64 - 2^10
      w.push_back((uint64_t)std::llrint(std::ldexp(b[0], s)));
      w.push_back((uint64_t)std::llrint(std::ldexp(b[1], s)));
      w.push_back(((uint64_t)q & ~63ull) | (uint64_t)sh);
      uint64_t amplitude;
      std::memcpy(&amplitude, &b[3], 8);
      w.push_back(amplitude);
    }
    if (fits) {
      prm[0] = word((uint64_t)(w.size() / 4));
      for (size_t k = 0; k < w.size(); ++k) prm[1 + k] = word(w[k]);
      return 100;
    }
    for (int k = 0; k < K; ++k) prm[1 + 4 * k + 2] = -1.0 / (2.0 * p[1 + 4 * k + 2] * p[1 + 4 * k + 2]);
    return f.kind;
  }
  if (f.kind == HDG_FIELD_FOURIER || f.kind == HDG_FIELD_EXP_FOURIER) {
    double kmax = 0.0, ksum = 0.0, asum = 0.0;
    bool fits = usable;
    for (int k = 0; k < K; ++k) {
      const double* b = &p[2 + 4 * k];
      fits = fits && std::isfinite(b[0]) && std::isfinite(b[1]) && std::isfinite(b[2]) && std::isfinite(b[3]);
      kmax = std::max(kmax, std::max(std::fabs(b[0]), std::fabs(b[1])));
      ksum = std::max(ksum, std::fabs(b[0]) + std::fabs(b[1]));
      asum += std::fabs(b[3]);
    }
    // the grid moves a phase by pi 2^-s (|kx| + |ky|) at most: no more than FP64's rounding of a phase of one turn, 2^-51
    if (!fits || !(asum < 1e300) || !(ksum <= std::ldexp(1.0 / 3.141592653589793, s - 51))) return f.kind;
    // wave numbers to 2^-60 of the largest, or to where the shift ends: 2^-123 of a turn over the domain
    const int u = std::min(kmax > 0.0 ? 60 - ceil_log2(kmax) : 60, 184 - s);
    const int w = asum > 0.0 ? 62 - ceil_log2(asum) : 0;
    const int sh = s + u - 64;
    if (sh < 0 || sh > 120 || w < -900 || w > 900) return f.kind;
    prm[0] = word((uint64_t)(uint32_t)K | ((uint64_t)sh << 32) | ((uint64_t)(uint16_t)(int16_t)w << 48));
    for (int k = 0; k < K; ++k) {
      const double* b = &p[2 + 4 * k];
      long double t = (long double)b[2] / 6.28318530717958647692528676655900577L;
      t -= std::floor(t);
      prm[2 + 4 * k] = word((uint64_t)std::llrint(std::ldexp(b[0], u)));
      prm[2 + 4 * k + 1] = word((uint64_t)std::llrint(std::ldexp(b[1], u)));
      prm[2 + 4 * k + 2] = word(t < 1.0L ? (uint64_t)(t * 18446744073709551616.0L) : 0ull);
      prm[2 + 4 * k + 3] = word((uint64_t)std::llrint(std::ldexp(b[3], w)));
    }
    return f.kind == HDG_FIELD_FOURIER ? 101 : 102;
  }
  return f.kind;
}

extern "C++" void populate_pages(void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
  if (!p || bytes == 0) return;
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = (uintptr_t)p & ~(page - 1);
  const int err = errno;
  madvise((void*)a, (uintptr_t)p + bytes - a, MADV_POPULATE_WRITE);
  errno = err;
#else
  (void)p;
  (void)bytes;
#endif
}

extern "C++" void ensure_fixed_fields(hdg_system* s, bool wait) {
  const std::vector<double>& xy = s->space->mesh->prob_xy_max;
  const int np = s->nprob;
  // magnitudes beyond which a product of the evaluation could leave FP64's range: the plain form
  constexpr int E_MIN = -400, E_MAX = 400;
  std::vector<int> ex(np);
  for (int P = 0; P < np; ++P) ex[P] = xy[P] > 0.0 && std::isfinite(xy[P]) ? coordinate_exponent(xy[P]) : E_MAX + 1;
  if (ex == s->fix_exp) return;
  std::vector<int> sc(np);
  std::vector<char> usable(np);
  std::vector<double> scale(np);
  for (int P = 0; P < np; ++P) {
    const int top = std::max(fixed_exponent(ex[P], s->fsp[P]), fixed_exponent(ex[P], s->ksp[P]));
    usable[P] = top >= E_MIN && top <= E_MAX;
    sc[P] = usable[P] ? 61 - top : 0;
    scale[P] = std::ldexp(1.0, sc[P]);
  }
  std::vector<double> all(scale);
  std::vector<int32_t> ints;
  for (auto* v : {&s->fsp, &s->ksp}) {
    std::vector<int32_t> off(np);
    for (int P = 0; P < np; ++P) {
      const FieldSpec& f = (*v)[P];
      const size_t at = all.size();
      off[P] = (int32_t)(at - np);
      all.insert(all.end(), f.prm.begin(), f.prm.end());
      ints.push_back(prepare_fixed(f, sc[P], ex[P], usable[P], all.data() + at));
    }
    ints.insert(ints.end(), off.begin(), off.end());
  }
  s->fix_ints = all.size();
  all.resize(all.size() + (ints.size() + 1) / 2);
  std::memcpy(&all[s->fix_ints], ints.data(), ints.size() * sizeof(int32_t));
  s->d_fix.upload(all.data(), all.size(), s->ctx->stream);
  if (wait) HDG_CUDA(cudaStreamSynchronize(s->ctx->stream));
  s->fix_exp = ex;
}

// ---------------------------------------------------------------- assembly
// Per-problem coefficients: f[P], kappa[P] (fields, or NULL), tau[P]; kappa_cell over all cells.
static void set_coefficients_many(hdg_system* s, const double* taus, const hdg_field* const* f,
                                  const hdg_field* const* kappa, const double* kappa_cell) {
  cudaStream_t st = s->ctx->stream;
  const int np = s->nprob;
  s->fsp.assign(np, FieldSpec());
  s->ksp.assign(np, FieldSpec());
  s->taus.assign(np, 1.0);
  std::vector<int32_t> fk(np), fo(np), kk(np), ko(np);
  std::vector<double> fp, kp;
  s->kappa_field = false;
  for (int P = 0; P < np; ++P) {
    s->taus[P] = taus ? taus[P] : 1.0;
    if (!(s->taus[P] > 0.0)) throw HdgError{HDG_ERR_ARG, "tau must be positive"};
    s->fsp[P] = field_from(f ? f[P] : nullptr, 0.0);
    s->ksp[P] = field_from(kappa ? kappa[P] : nullptr, 1.0);
    if (kappa && kappa[P]) s->kappa_field = true;
    fk[P] = s->fsp[P].kind;
    fo[P] = (int32_t)fp.size();
    fp.insert(fp.end(), s->fsp[P].prm.begin(), s->fsp[P].prm.end());
    kk[P] = s->ksp[P].kind;
    ko[P] = (int32_t)kp.size();
    kp.insert(kp.end(), s->ksp[P].prm.begin(), s->ksp[P].prm.end());
  }
  s->d_fkind.upload(fk.data(), np, st);
  s->d_foff.upload(fo.data(), np, st);
  s->d_fprm.upload(fp.data(), fp.size(), st);
  // the element kernels evaluate a Gaussian bump as a exp(|x - c|^2 k) with k = -1/(2 s^2) formed
  // here once, instead of dividing by 2 s^2 at every quadrature point
  std::vector<double> fpp(fp);
  for (int P = 0; P < np; ++P)
    if (fk[P] == HDG_FIELD_BUMPS) {
      const int K = (int)fpp[fo[P]];
      for (int b = 0; b < K; ++b) {
        double& sw = fpp[fo[P] + 1 + 4 * b + 2];
        sw = -1.0 / (2.0 * sw * sw);
      }
    }
  s->d_fprep.upload(fpp.data(), fpp.size(), st);
  s->fix_exp.clear();  // the fixed-point form is of the old fields
  s->d_kkind.upload(kk.data(), np, st);
  s->d_koff.upload(ko.data(), np, st);
  s->d_kprm.upload(kp.data(), kp.size(), st);
  s->d_tau.upload(s->taus.data(), np, st);
  s->tau = s->taus[0];
  s->kappa_cells = kappa_cell != nullptr;
  if (kappa_cell) {
    for (int c = 0; c < s->nc; ++c)
      if (!(kappa_cell[c] > 0.0)) throw HdgError{HDG_ERR_ARG, "kappa must be positive"};
    s->d_kappa.upload(kappa_cell, (size_t)s->nc, st);
  }
  ensure_fixed_fields(s, false);
  HDG_CUDA(cudaStreamSynchronize(st));  // the host staging vectors go out of scope
}

// The same source, coefficient and tau for every problem of the system.
static void set_coefficients(hdg_system* s, double tau, const hdg_field* f, const hdg_field* kappa,
                             const double* kappa_cell) {
  std::vector<const hdg_field*> fs(s->nprob, f), ks(s->nprob, kappa);
  std::vector<double> ts(s->nprob, tau);
  set_coefficients_many(s, ts.data(), fs.data(), kappa ? ks.data() : nullptr, kappa_cell);
}

extern "C++" void assemble_async(hdg_system* s, cudaStream_t st) {
  const bool prof = s->ctx->profiling;
  HDG_CUDA(cudaMemsetAsync(s->d_scal.p, 0, 4 * sizeof(double), st));
  if (prof) s->ev_element.start(st);
  launch_element_condense(s, st);
  if (prof) {
    s->ev_element.stop(st);
    s->ev_gather.start(st);
  }
  launch_gather(s, st);
  if (prof) s->ev_gather.stop(st);
  s->applied = false;
  s->have_solution = false;
  s->have_recovery = false;
}

extern "C++" void assembly_check(hdg_system* s, cudaStream_t st) {
  double sc[2];
  HDG_CUDA(cudaMemcpyAsync(sc, s->d_scal.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  HDG_CUDA(cudaStreamSynchronize(st));
  int err = 0;
  std::memcpy(&err, &sc[1], sizeof(int));
  if (err & 1) throw HdgError{HDG_ERR_NEG_DETJ, "det(J) is not positive on some cell"};
  if (err & 2) throw HdgError{HDG_ERR_SINGULAR, "a local system has a zero pivot (singular)"};
}

static void assemble_now(hdg_system* s) {
  assemble_async(s, s->ctx->stream);
  assembly_check(s, s->ctx->stream);
}

static int assemble_condense_impl(hdg_space* space, double tau, const hdg_field* f, const hdg_field* kappa,
                                  const double* kappa_cell, int precision, const double* taus_many,
                                  const hdg_field* const* fields_many, const hdg_field* const* kappas_many,
                                  hdg_system** out) {
  if (!space || !out) return HDG_ERR_ARG;
  hdg_ctx* ctx = space->mesh->ctx;
  if (!fields_many && !(tau > 0.0)) return fail(ctx, HDG_ERR_ARG, "tau must be positive");
  if (precision != HDG_PREC_FP64 && precision != HDG_PREC_MIXED) return fail(ctx, HDG_ERR_ARG, "bad precision");
  return guard(ctx, [&]() -> int {
    set_device(ctx);
    hdg_system* s = new hdg_system();
    try {
      s->space = space;
      s->ctx = ctx;
      s->precision = precision;
      s->he_tau = space->he_tau;
      s->amg_tune_time = g_tuning_allowed;
      const RefTables& t = space->t;
      s->nw = t.nw;
      s->nt = t.nt;
      s->n = 3 * t.nw;
      s->m = 3 * t.nt;
      s->nc = space->mesh->nc;
      s->nf = space->mesh->nf;
      s->ndofs = s->nf * s->nt;
      s->nprob = space->mesh->nprob;
      if (fields_many) set_coefficients_many(s, taus_many, fields_many, kappas_many, kappa_cell);
      else set_coefficients(s, tau, f, kappa, kappa_cell);
      s->d_AB.alloc((size_t)s->nc * s->m * (s->m + 1));
      s->d_KB.alloc((size_t)s->nc * s->n * (s->m + 1));
      s->d_scal.alloc(4);
      build_block_structure(s);
      build_segments(s);
      s->d_val.alloc((size_t)hdg_system::SLOTS * s->nt * s->ndofs);
      s->d_b.alloc((size_t)s->ndofs);
      assemble_now(s);
    } catch (...) {
      delete s;
      throw;
    }
    *out = s;
    return HDG_OK;
  });
}

int hdg_assemble_condense(hdg_space* space, double tau, const hdg_field* f, const hdg_field* kappa,
                          const double* kappa_cell, int precision, hdg_system** out) {
  return assemble_condense_impl(space, tau, f, kappa, kappa_cell, precision, nullptr, nullptr, nullptr, out);
}

int hdg_assemble_condense_batch(hdg_space* space, const double* tau, const hdg_field* f, const hdg_field* kappa,
                                const double* kappa_cell, int precision, hdg_system** out) {
  if (!space || !f || !out) return HDG_ERR_ARG;
  const int np = space->mesh->nprob;
  std::vector<const hdg_field*> fs(np), ks(np);
  for (int P = 0; P < np; ++P) {
    fs[P] = &f[P];
    ks[P] = kappa ? &kappa[P] : nullptr;
  }
  return assemble_condense_impl(space, 1.0, nullptr, nullptr, kappa_cell, precision, tau, fs.data(),
                                kappa ? ks.data() : nullptr, out);
}

int hdg_system_reassemble_batch(hdg_system* s, const double* tau, const hdg_field* f, const hdg_field* kappa,
                                const double* kappa_cell) {
  if (!s || !f) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    std::vector<const hdg_field*> fs(s->nprob), ks(s->nprob);
    for (int P = 0; P < s->nprob; ++P) {
      fs[P] = &f[P];
      ks[P] = kappa ? &kappa[P] : nullptr;
    }
    set_coefficients_many(s, tau, fs.data(), kappa ? ks.data() : nullptr, kappa_cell);
    assemble_now(s);
    return HDG_OK;
  });
}

int hdg_system_reassemble(hdg_system* s, double tau, const hdg_field* f, const hdg_field* kappa,
                          const double* kappa_cell) {
  if (!s) return HDG_ERR_ARG;
  if (!(tau > 0.0)) return fail(s->ctx, HDG_ERR_ARG, "tau must be positive");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    set_coefficients(s, tau, f, kappa, kappa_cell);
    assemble_now(s);
    return HDG_OK;
  });
}

int hdg_system_reassemble_resident(hdg_system* s) {
  if (!s) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    assemble_now(s);
    return HDG_OK;
  });
}

int hdg_system_sizes(const hdg_system* s, int* ndofs, int64_t* nnz, int* n, int* m) {
  if (!s) return HDG_ERR_ARG;
  if (ndofs) *ndofs = s->ndofs;
  if (nnz) *nnz = s->nnz;
  if (n) *n = s->n;
  if (m) *m = s->m;
  return HDG_OK;
}

int hdg_system_get_csc(const hdg_system* s, int base, int64_t* colptr, int64_t* rowval, double* nzval, double* rhs) {
  if (!s || (base != 0 && base != 1)) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    run_export_csc(s, base, colptr, rowval, nzval, rhs, s->ctx->stream);
    return HDG_OK;
  });
}

int hdg_system_get_element_blocks(const hdg_system* s, double* Ate, double* bte, double* Ke, double* be) {
  if (!s) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    cudaStream_t st = s->ctx->stream;
    const int n = s->n, m = s->m, nc = s->nc;
    std::vector<double> AB((size_t)nc * m * (m + 1)), KB((size_t)nc * n * (m + 1));
    if (Ate || bte) s->d_AB.download(AB.data(), AB.size(), st);
    if ((Ke || be) && s->kb_u_only) {  // the element path kept the u rows only: form the q rows
      DevBuf<double> full;
      full.alloc(KB.size());
      launch_expand_ke(const_cast<hdg_system*>(s), full.p, st);
      full.download(KB.data(), KB.size(), st);
      HDG_CUDA(cudaStreamSynchronize(st));
    } else if (Ke || be) {
      s->d_KB.download(KB.data(), KB.size(), st);
    }
    HDG_CUDA(cudaStreamSynchronize(st));
    for (int c = 0; c < nc; ++c) {
      for (int i = 0; i < m; ++i) {
        const double* r = &AB[((size_t)c * m + i) * (m + 1)];
        if (Ate) std::memcpy(Ate + ((size_t)c * m + i) * m, r, m * sizeof(double));
        if (bte) bte[(size_t)c * m + i] = r[m];
      }
      for (int i = 0; i < n; ++i) {
        const double* r = &KB[((size_t)c * n + i) * (m + 1)];
        if (Ke) std::memcpy(Ke + ((size_t)c * n + i) * m, r, m * sizeof(double));
        if (be) be[(size_t)c * n + i] = r[m];
      }
    }
    return HDG_OK;
  });
}

// ---------------------------------------------------------------- Dirichlet
int hdg_dirichlet(const hdg_space* sp, const char* faceset, const hdg_field* g, int32_t* dofs, double* vals,
                  int* count) {
  if (!sp || !faceset || !count) return HDG_ERR_ARG;
  const hdg_mesh* m = sp->mesh;
  auto it = m->facesets.find(faceset);
  if (it == m->facesets.end()) return fail(m->ctx, HDG_ERR_UNKNOWN_SET, std::string("no face set ") + faceset);
  const RefTables& t = sp->t;
  const int nt = t.nt, nfq = t.nfq;
  *count = (int)it->second.size() * nt;
  if (!dofs && !vals) return HDG_OK;
  std::string why;
  if (field_check(g, &why) != HDG_OK) return fail(m->ctx, HDG_ERR_ARG, why);
  FieldSpec gs = field_from(g, 0.0);
  static const double EDGE[3][4] = {{1, 0, 0, 1}, {0, 1, 0, 0}, {0, 0, 1, 0}};
  static const int EN[3][2] = {{1, 2}, {2, 0}, {0, 1}};
  int k = 0;
  // faces in increasing id (the reference loops 1:getnfaces and tests membership)
  for (int32_t f : it->second) {
    if (m->faces[4 * f + 3] >= 0) return fail(m->ctx, HDG_ERR_NOT_BOUNDARY, "Face " + std::to_string(f + 1) + " is not in boundary");
    const int c = m->faces[4 * f + 2];
    int fl = 0;
    while (m->cfaces[3 * c + fl] != f) ++fl;
    const bool o = m->cells[3 * c + EN[fl][1]] > m->cells[3 * c + EN[fl][0]];
    // the reference's projection (src/boundary.jl:27-37): the accumulator N runs across the
    // basis functions of a face, the weights are the parent's volume weights, no |e|
    double acc = 0.0;
    for (int i = 0; i < nt; ++i) {
      for (int q = 0; q < nfq; ++q) {
        const int oq = o ? q : nfq - 1 - q;
        const double s = t.fx[oq];
        const double ex = (1.0 - s) * EDGE[fl][0] + s * EDGE[fl][2], ey = (1.0 - s) * EDGE[fl][1] + s * EDGE[fl][3];
        const double L[3] = {1.0 - ex - ey, ex, ey};
        double xq = 0, yq = 0;
        for (int a = 0; a < 3; ++a) {
          xq += L[a] * m->xy[2 * m->cells[3 * c + a]];
          yq += L[a] * m->xy[2 * m->cells[3 * c + a] + 1];
        }
        acc += t.qw[q] * eval_field_host(gs, xq, yq) * t.T[i * nfq + q];
      }
      if (vals) vals[k] = acc;
      if (dofs) dofs[k] = f * nt + i + 1;
      ++k;
    }
  }
  return HDG_OK;
}

int hdg_dirichlet_l2(const hdg_space* sp, const char* faceset, const hdg_field* g, int32_t* dofs, double* vals,
                     int* count) {
  if (!sp || !faceset || !count) return HDG_ERR_ARG;
  const hdg_mesh* m = sp->mesh;
  auto it = m->facesets.find(faceset);
  if (it == m->facesets.end()) return fail(m->ctx, HDG_ERR_UNKNOWN_SET, std::string("no face set ") + faceset);
  const RefTables& t = sp->t;
  const int nt = t.nt, nfq = t.nfq;
  *count = (int)it->second.size() * nt;
  if (!dofs && !vals) return HDG_OK;
  std::string why;
  if (field_check(g, &why) != HDG_OK) return fail(m->ctx, HDG_ERR_ARG, why);
  FieldSpec gs = field_from(g, 0.0);
  static const double EDGE[3][4] = {{1, 0, 0, 1}, {0, 1, 0, 0}, {0, 0, 1, 0}};
  static const int EN[3][2] = {{1, 2}, {2, 0}, {0, 1}};
  int k = 0;
  for (int32_t f : it->second) {
    if (m->faces[4 * f + 3] >= 0) return fail(m->ctx, HDG_ERR_NOT_BOUNDARY, "Face " + std::to_string(f + 1) + " is not in boundary");
    const int c = m->faces[4 * f + 2];
    int fl = 0;
    while (m->cfaces[3 * c + fl] != f) ++fl;
    const bool o = m->cells[3 * c + EN[fl][1]] > m->cells[3 * c + EN[fl][0]];
    // L2 projection onto the face's orthonormal Legendre basis: u_i = int_0^1 g mu_i ds (the
    // face length cancels against the trace mass matrix |e| I), with the face rule's weights
    for (int i = 0; i < nt; ++i) {
      double acc = 0.0;
      for (int q = 0; q < nfq; ++q) {
        const int oq = o ? q : nfq - 1 - q;
        const double s = t.fx[oq];
        const double ex = (1.0 - s) * EDGE[fl][0] + s * EDGE[fl][2], ey = (1.0 - s) * EDGE[fl][1] + s * EDGE[fl][3];
        const double L[3] = {1.0 - ex - ey, ex, ey};
        double xq = 0, yq = 0;
        for (int a = 0; a < 3; ++a) {
          xq += L[a] * m->xy[2 * m->cells[3 * c + a]];
          yq += L[a] * m->xy[2 * m->cells[3 * c + a] + 1];
        }
        acc += t.fw[q] * eval_field_host(gs, xq, yq) * t.T[i * nfq + q];
      }
      if (vals) vals[k] = acc;
      if (dofs) dofs[k] = f * nt + i + 1;
      ++k;
    }
  }
  return HDG_OK;
}

int hdg_space_set_he_tau(hdg_space* sp, int on) {
  if (!sp) return HDG_ERR_ARG;
  sp->he_tau = on != 0;
  return HDG_OK;
}

// Validates a Dirichlet set, records its faces for the multigrid setup (a new set invalidates the
// symbolic part) and scatters it on the device.
static void set_dirichlet_now(hdg_system* s, const int32_t* dofs, const double* vals, int n) {
  std::vector<int32_t> d0(n);
  std::vector<double> v(vals, vals + n);
  for (int k = 0; k < n; ++k) {
    if (dofs[k] < 1 || dofs[k] > s->ndofs) throw HdgError{HDG_ERR_ARG, "prescribed dof out of range"};
    d0[k] = dofs[k] - 1;
  }
  // prescribed faces (all their dofs are prescribed together): the multigrid setup leaves them
  // out of its aggregates
  std::vector<char> dir(s->nf, 0);
  for (int k = 0; k < n; ++k) dir[d0[k] / s->nt] = 1;
  if (dir != s->h_dir_face && s->amg) {
    destroy_amg(s->amg);
    s->amg = nullptr;
  }
  s->h_dir_face.swap(dir);
  launch_dirichlet_scatter(s, d0, v, s->ctx->stream);
}

int hdg_apply_dirichlet(hdg_system* s, const int32_t* dofs, const double* vals, int n) {
  if (!s || n < 0 || (n > 0 && (!dofs || !vals))) return HDG_ERR_ARG;
  if (s->applied) return fail(s->ctx, HDG_ERR_ARG, "apply! was already called on this system");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    if (s->ctx->profiling) s->ev_apply.start(s->ctx->stream);
    set_dirichlet_now(s, dofs, vals, n);
    launch_dirichlet_apply(s, s->ctx->stream);
    if (s->ctx->profiling) s->ev_apply.stop(s->ctx->stream);
    s->applied = true;
    return HDG_OK;
  });
}

int hdg_system_set_dirichlet(hdg_system* s, const int32_t* dofs, const double* vals, int n) {
  if (!s || n < 0 || (n > 0 && (!dofs || !vals))) return HDG_ERR_ARG;
  // allowed on an applied system: the set takes effect at the next apply!, which needs a
  // reassembly first (hdg_batch_step refuses HDG_STEP_APPLY without HDG_STEP_ASSEMBLE there)
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    set_dirichlet_now(s, dofs, vals, n);
    return HDG_OK;
  });
}

int hdg_system_set_coefficients_batch(hdg_system* s, const double* tau, const hdg_field* f, const hdg_field* kappa,
                                      const double* kappa_cell) {
  if (!s || !f) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    std::vector<const hdg_field*> fs(s->nprob), ks(s->nprob);
    for (int P = 0; P < s->nprob; ++P) {
      fs[P] = &f[P];
      ks[P] = kappa ? &kappa[P] : nullptr;
    }
    set_coefficients_many(s, tau, fs.data(), kappa ? ks.data() : nullptr, kappa_cell);
    return HDG_OK;
  });
}

// ---------------------------------------------------------------- solve / recover
static hdg_solver solver_defaults(const hdg_solver* o) {
  hdg_solver d{1e-12, 100000, HDG_PREC_FP64, 32, 1e-5, HDG_PRECOND_JACOBI};
  if (!o) return d;
  hdg_solver r = *o;
  if (!(r.tol > 0)) r.tol = d.tol;
  if (r.maxit <= 0) r.maxit = d.maxit;
  if (r.chunk <= 0) r.chunk = d.chunk;
  if (!(r.inner_tol > 0)) r.inner_tol = d.inner_tol;
  if (r.preconditioner != HDG_PRECOND_AMG) r.preconditioner = HDG_PRECOND_JACOBI;
  return r;
}

int hdg_solve(hdg_system* s, const hdg_solver* opts, double* uhat, hdg_stats* stats) {
  if (!s) return HDG_ERR_ARG;
  if (!s->applied) return fail(s->ctx, HDG_ERR_ARG, "apply the Dirichlet conditions (hdg_apply_dirichlet) first");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    hdg_solver o = solver_defaults(opts);
    int rc = run_solve(s, o, stats);
    s->have_solution = (rc == HDG_OK || rc == HDG_ERR_NO_CONVERGENCE);
    if (uhat && s->have_solution) {
      s->d_x.download(uhat, (size_t)s->ndofs, s->ctx->stream);
      HDG_CUDA(cudaStreamSynchronize(s->ctx->stream));
    }
    if (rc == HDG_ERR_NO_CONVERGENCE) return fail(s->ctx, rc, "CG did not reach the tolerance within maxit");
    if (rc == HDG_ERR_BREAKDOWN) return fail(s->ctx, rc, "CG breakdown: the trace system is not definite");
    return rc;
  });
}

int hdg_refine(hdg_system* s, const hdg_solver* opts, int steps, double correction_tol, double* uhat,
               hdg_stats* stats) {
  if (!s) return HDG_ERR_ARG;
  if (!s->have_solution) return fail(s->ctx, HDG_ERR_ARG, "solve first (hdg_solve)");
  if (steps < 0 || steps > 16) return fail(s->ctx, HDG_ERR_ARG, "refinement steps must be in [0, 16]");
  if (!(correction_tol > 0.0) || !(correction_tol < 1.0))
    return fail(s->ctx, HDG_ERR_ARG, "the correction tolerance must lie in (0, 1)");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    hdg_solver o = solver_defaults(opts);
    std::vector<hdg_stats> per;
    int rc = run_refine(s, o, steps, correction_tol, &per);
    if (stats) {
      hdg_stats agg{0, steps, 0.0, 1};
      for (auto& r : per) {
        agg.iterations = std::max(agg.iterations, r.iterations);
        agg.rel_residual = std::max(agg.rel_residual, r.rel_residual);
        agg.converged = agg.converged && r.converged;
      }
      *stats = agg;
    }
    if (uhat) {
      s->d_x.download(uhat, (size_t)s->ndofs, s->ctx->stream);
      HDG_CUDA(cudaStreamSynchronize(s->ctx->stream));
    }
    if (rc == HDG_ERR_NO_CONVERGENCE) return fail(s->ctx, rc, "a correction solve did not reach its tolerance");
    if (rc == HDG_ERR_BREAKDOWN) return fail(s->ctx, rc, "CG breakdown in a correction solve");
    return rc;
  });
}

int hdg_recover_into(hdg_system* s, double* q, double* u, double* uhat_cell, int by_function) {
  if (!s) return HDG_ERR_ARG;
  if (!s->have_solution) return fail(s->ctx, HDG_ERR_ARG, "solve first");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    cudaStream_t st = s->ctx->stream;
    if (s->ctx->profiling) s->ev_recover.start(st);
    launch_recover(s, st);
    if (s->ctx->profiling) s->ev_recover.stop(st);
    s->have_recovery = true;
    // the three arrays are laid out on the device and copied straight to the caller's: through a host staging vector,
    // a host loop per cell and a second copy, 2*512^2 cells of p = 3 took 36 ms.  In pieces of 32 MB, whatever the system.
    if (q || u || uhat_cell) {
      const size_t per_cell = sizeof(double) * ((q ? 2 * s->nw : 0) + (u ? s->nw : 0) + (uhat_cell ? s->m : 0));
      const int piece = (int)std::min<size_t>(s->nc, std::max<size_t>(1, (size_t(32) << 20) / per_cell));
      DevBuf<double> dq, du, dx;
      struct Part {
        double* to;
        DevBuf<double>* from;
        int width;
      };
      const Part parts[3] = {{q, &dq, 2 * s->nw}, {u, &du, s->nw}, {uhat_cell, &dx, s->m}};
      for (const Part& p : parts)
        if (p.to) p.from->alloc((size_t)piece * p.width);
      for (int c0 = 0; c0 < s->nc; c0 += piece) {
        const int c1 = std::min(s->nc, c0 + piece);
        launch_recover_split(s, c0, c1, dq.p, du.p, dx.p, by_function != 0, st);
        for (const Part& p : parts)
          if (p.to) populate_pages(p.to + (size_t)c0 * p.width, sizeof(double) * (size_t)(c1 - c0) * p.width);
        for (const Part& p : parts)
          if (p.to) p.from->download(p.to + (size_t)c0 * p.width, (size_t)(c1 - c0) * p.width, st);
      }
      HDG_CUDA(cudaStreamSynchronize(st));
    }
    return HDG_OK;
  });
}

int hdg_recover(hdg_system* s, double* q, double* u, double* uhat_cell) {
  return hdg_recover_into(s, q, u, uhat_cell, 0);
}

int hdg_errornorm_l2sq(hdg_system* s, const hdg_field* uex, double* out) {
  if (!s || !uex || !out) return HDG_ERR_ARG;
  if (!s->have_recovery) return fail(s->ctx, HDG_ERR_ARG, "recover first");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    *out = run_errornorm(s, field_from(uex, 0.0), s->ctx->stream);
    return HDG_OK;
  });
}

int hdg_nodal_avg(hdg_system* s, double* out) {
  if (!s || !out) return HDG_ERR_ARG;
  if (!s->have_recovery) return fail(s->ctx, HDG_ERR_ARG, "recover first");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    run_nodal_avg(s, out, s->ctx->stream);
    return HDG_OK;
  });
}

int hdg_system_timings(hdg_system* s, hdg_timings* out) {
  if (!s || !out) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    std::memset(out, 0, sizeof(*out));
    out->element_ms = s->ev_element.ms();
    out->gather_ms = s->ev_gather.ms();
    out->apply_ms = s->ev_apply.ms();
    out->cg_ms = s->ev_cg.ms();
    out->recover_ms = s->ev_recover.ms();
    double ta = 0, tb = 0;
    for (auto* e : s->ev_cg_a) ta += e->ms();
    for (auto* e : s->ev_cg_b) tb += e->ms();
    out->cg_samples = (int)s->ev_cg_a.size();
    if (out->cg_samples) {
      out->cg_a_ms = ta / out->cg_samples;
      out->cg_b_ms = tb / out->cg_samples;
      out->cg_a_bytes = s->prof_a_bytes / out->cg_samples;
      out->cg_b_bytes = s->prof_b_bytes / out->cg_samples;
    }
    if (s->prof_res_iters > 0) {  // resident iteration: one launch makes many, both phases in it
      double tr = 0;
      for (auto* e : s->ev_res) tr += e->ms();
      out->cg_samples = (int)s->prof_res_iters;
      out->cg_a_ms = tr / (double)s->prof_res_iters;
      out->cg_b_ms = 0;
      out->cg_a_bytes = s->prof_all_bytes / (double)s->prof_res_iters;
      out->cg_b_bytes = 0;
    }
    out->cg_iterations = s->cg_iterations;
    out->cg_bytes = s->prof_all_bytes;
    return HDG_OK;
  });
}

int hdg_system_kernel_sample(hdg_system* s, int which, double* total_ms, double* total_bytes, int* launches) {
  if (!s || !total_ms || !total_bytes || !launches) return HDG_ERR_ARG;
  if (which != HDG_SAMPLE_CHEB0 && which != HDG_SAMPLE_L1SWEEP)
    return fail(s->ctx, HDG_ERR_ARG, "unknown kernel sample");
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    const std::vector<EventPair*>& ev = which == HDG_SAMPLE_CHEB0 ? s->ev_cheb0 : s->ev_l1;
    double t = 0.0;
    for (auto* e : ev) t += e->ms();
    *total_ms = t;
    *total_bytes = which == HDG_SAMPLE_CHEB0 ? s->prof_cheb0_bytes : s->prof_l1_bytes;
    *launches = (int)ev.size();
    return HDG_OK;
  });
}

int hdg_system_destroy(hdg_system* s) {
  if (s) {
    cudaSetDevice(s->ctx->device);
    cudaStreamSynchronize(s->ctx->stream);
    delete s;
  }
  return HDG_OK;
}

int hdg_solve_batch(int nsys, hdg_system* const* systems, const hdg_solver* opts, hdg_stats* stats) {
  if (nsys < 1 || !systems) return HDG_ERR_ARG;
  hdg_ctx* ctx = systems[0]->ctx;
  for (int i = 0; i < nsys; ++i) {
    if (!systems[i]) return HDG_ERR_ARG;
    if (!systems[i]->applied) return fail(systems[i]->ctx, HDG_ERR_ARG, "apply the Dirichlet conditions first");
  }
  return guard(ctx, [&]() -> int {
    set_device(ctx);
    hdg_solver o = solver_defaults(opts);
    std::vector<hdg_system*> v(systems, systems + nsys);
    std::vector<std::vector<hdg_stats>> st;
    int rc = run_solve_many(v, o, &st);
    size_t k = 0;
    for (int i = 0; i < nsys; ++i) {
      v[i]->have_solution = (rc == HDG_OK || rc == HDG_ERR_NO_CONVERGENCE);
      for (auto& r : st[i]) {
        if (stats) stats[k] = r;
        ++k;
      }
    }
    if (rc == HDG_ERR_NO_CONVERGENCE) return fail(ctx, rc, "some problem did not reach the tolerance within maxit");
    if (rc == HDG_ERR_BREAKDOWN) return fail(ctx, rc, "CG breakdown in some problem");
    return rc;
  });
}

int hdg_host_alloc(size_t bytes, void** out) {
  if (!out) return HDG_ERR_ARG;
  *out = nullptr;
  if (bytes == 0) return HDG_OK;
  return cudaMallocHost(out, bytes) == cudaSuccess ? HDG_OK : HDG_ERR_OOM;
}

int hdg_host_free(void* p) {
  if (p) cudaFreeHost(p);
  return HDG_OK;
}

int hdg_system_set_download(hdg_system* s, double* uhat, double* qu) {
  if (!s) return HDG_ERR_ARG;
  s->h_dl_uhat = uhat;
  s->h_dl_qu = qu;
  return HDG_OK;
}

int hdg_batch_step(int nsys, hdg_system* const* systems, const hdg_solver* opts, int flags, hdg_stats* stats) {
  if (nsys < 1 || !systems ||
      (flags & ~(HDG_STEP_ASSEMBLE | HDG_STEP_APPLY | HDG_STEP_RECOVER | HDG_STEP_DOWNLOAD)))
    return HDG_ERR_ARG;
  hdg_ctx* ctx = systems[0] ? systems[0]->ctx : nullptr;
  if (!ctx) return HDG_ERR_ARG;
  for (int i = 0; i < nsys; ++i) {
    hdg_system* s = systems[i];
    if (!s || s->ctx != ctx) return fail(ctx, HDG_ERR_ARG, "the systems of a step must share one context");
    for (int j = 0; j < i; ++j)
      if (systems[j] == s) return fail(ctx, HDG_ERR_ARG, "a system appears twice in the step");
    if ((flags & HDG_STEP_DOWNLOAD) && s->h_dl_qu && !(flags & HDG_STEP_RECOVER))
      return fail(ctx, HDG_ERR_ARG, "downloading (q, u) needs HDG_STEP_RECOVER");
    if (flags & HDG_STEP_APPLY) {
      if (!s->dir_ready) return fail(ctx, HDG_ERR_ARG, "no Dirichlet set recorded (hdg_system_set_dirichlet)");
      if (s->applied && !(flags & HDG_STEP_ASSEMBLE))
        return fail(ctx, HDG_ERR_ARG, "apply! was already called on this system");
    } else {
      if (flags & HDG_STEP_ASSEMBLE) return fail(ctx, HDG_ERR_ARG, "assembly undoes apply!: add HDG_STEP_APPLY");
      if (!s->applied) return fail(ctx, HDG_ERR_ARG, "apply the Dirichlet conditions first");
    }
  }
  return guard(ctx, [&]() -> int {
    set_device(ctx);
    hdg_solver o = solver_defaults(opts);
    std::vector<hdg_system*> v(systems, systems + nsys);
    std::vector<std::vector<hdg_stats>> st;
    int rc = run_batch_step(v, o, flags, &st);
    size_t k = 0;
    for (int i = 0; i < nsys; ++i) {
      v[i]->have_solution = (rc == HDG_OK || rc == HDG_ERR_NO_CONVERGENCE);
      v[i]->have_recovery = v[i]->have_solution && (flags & HDG_STEP_RECOVER);
      for (auto& r : st[i]) {
        if (stats) stats[k] = r;
        ++k;
      }
    }
    if (rc == HDG_ERR_NO_CONVERGENCE) return fail(ctx, rc, "some problem did not reach the tolerance within maxit");
    if (rc == HDG_ERR_BREAKDOWN) return fail(ctx, rc, "CG breakdown in some problem");
    return rc;
  });
}

int hdg_system_get_solution(const hdg_system* s, double* uhat, double* qu) {
  if (!s || !s->have_solution) return HDG_ERR_ARG;
  return guard(s->ctx, [&]() -> int {
    set_device(s->ctx);
    if (uhat) s->d_x.download(uhat, (size_t)s->ndofs, s->ctx->stream);
    if (qu) {
      if (!s->have_recovery) return fail(s->ctx, HDG_ERR_ARG, "recover first");
      s->d_qu.download(qu, (size_t)s->nc * s->n, s->ctx->stream);
    }
    HDG_CUDA(cudaStreamSynchronize(s->ctx->stream));
    return HDG_OK;
  });
}

int hdg_mesh_concat(hdg_ctx* ctx, int nparts, const hdg_mesh* const* parts, hdg_mesh** out) {
  if (!out || nparts < 1 || !parts) return fail(ctx, HDG_ERR_ARG, "hdg_mesh_concat: bad arguments");
  return guard(ctx, [&]() -> int {
    if (ctx) set_device(ctx);
    std::vector<const hdg_mesh*> v(parts, parts + nparts);
    for (auto* p : v)
      if (!p) return fail(ctx, HDG_ERR_ARG, "hdg_mesh_concat: null part");
    hdg_mesh* m = new hdg_mesh();
    m->ctx = ctx;
    try {
      mesh_concat(m, v);
      if (ctx) m->upload();
    } catch (...) {
      delete m;
      throw;
    }
    *out = m;
    return HDG_OK;
  });
}

int hdg_mesh_problems(const hdg_mesh* m, int* nprob, int32_t* node0, int32_t* cell0, int32_t* face0) {
  if (!m || !nprob) return HDG_ERR_ARG;
  *nprob = m->nprob;
  for (int P = 0; P <= m->nprob; ++P) {
    if (node0) node0[P] = m->prob_node0[P];
    if (cell0) cell0[P] = m->prob_cell0[P];
    if (face0) face0[P] = m->prob_face0[P];
  }
  return HDG_OK;
}

int hdg_solve_poisson(hdg_space* space, double tau, const hdg_field* f, const hdg_field* kappa,
                      const double* kappa_cell, const char* faceset, const hdg_field* g, const hdg_solver* opts,
                      double* uhat, double* q, double* u, hdg_stats* stats) {
  hdg_system* s = nullptr;
  int prec = opts ? opts->precision : HDG_PREC_FP64;
  int rc = hdg_assemble_condense(space, tau, f, kappa, kappa_cell, prec, &s);
  if (rc != HDG_OK) return rc;
  int cnt = 0;
  rc = hdg_dirichlet(space, faceset ? faceset : "boundary", g, nullptr, nullptr, &cnt);
  std::vector<int32_t> dofs(cnt);
  std::vector<double> vals(cnt);
  if (rc == HDG_OK) rc = hdg_dirichlet(space, faceset ? faceset : "boundary", g, dofs.data(), vals.data(), &cnt);
  if (rc == HDG_OK) rc = hdg_apply_dirichlet(s, dofs.data(), vals.data(), cnt);
  if (rc == HDG_OK) rc = hdg_solve(s, opts, uhat, stats);
  if (rc == HDG_OK) rc = hdg_recover(s, q, u, nullptr);
  hdg_system_destroy(s);
  return rc;
}

}  // extern "C"
