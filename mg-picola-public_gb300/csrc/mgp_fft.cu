// Power-of-two 3D transforms (N = 64 .. 1024) and the k-space passes fused into
// them: the host side of the kernels of mgp_fft.cuh.
//
// Passes of one PM step (grid = one padded N^3 grid of 4 N^3 bytes), each pass
// reading and writing its grids once:
//   density      z rows rho -> dk, y
//   LCDM         x: dk -> delta(k), and the two inverse transforms of the
//                force pass (1 grid read, 3 written)
//   screening    x: dk -> delta(k), and the filtered inverse (1 read, 2
//                written); y; z rows: inverse, screening, forward (2 read, 2
//                written); y; x: source spectrum and the force pass
//   forces       y: 2 grids read, 3 written; z rows of the three grids
// cuFFT's 3D plans need three read-write passes a transform and the k-space
// passes their own.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <vector>

#include "mgp_fft.h"
#include "mgp_internal.h"

#define RET_IF(x)                  \
  do {                             \
    int rc_ = (x);                 \
    if (rc_ != MGP_OK) return rc_; \
  } while (0)

static const mgp_fft_ops *ops_for(int N) {
  switch (N) {
    case 64: return mgp_fft_ops_64();
    case 128: return mgp_fft_ops_128();
    case 256: return mgp_fft_ops_256();
    case 512: return mgp_fft_ops_512();
    case 1024: return mgp_fft_ops_1024();
  }
  return NULL;
}

int mgp_fft_has(int N) { return ops_for(N) != NULL; }
// Whether the context's grids take these transforms.
int mgp_fft_supported(const mgp_ctx *c) { return mgp_fft_has(c->g.N); }

static int sms_of(const mgp_ctx *c) {
  int sms = 152;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  return sms;
}

static int launched(int rc) {
  if (rc) return mgp_set_error(MGP_ECUDA, "transform pass not available");
  MGP_CHECK_LAUNCH();
  g_kernel_launches++;
  return MGP_OK;
}

// A table to the device, there when the call returns (at context creation).
static int upload(mgp_ctx *c, float *dst, const void *src, size_t bytes) {
  MGP_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, c->stream));
  MGP_CUDA(cudaStreamSynchronize(c->stream));
  return MGP_OK;
}

// Twiddle tables of size N on the device: W_N^m (m < N), then the row passes'
// tables (mgp_fft.cuh, fft_row).
static int make_table(mgp_ctx *c, int N, float **out) {
  const mgp_fft_ops *o = ops_for(N);
  if (!o || *out) return MGP_OK;
  std::vector<float2> h;
  auto push = [&](double num, double den) {
    const double a = -2.0 * M_PI * num / den;
    h.push_back(make_float2((float)cos(a), (float)sin(a)));
  };
  for (int m = 0; m < N; m++) push(m, N);
  int ns = o->radix[0];
  for (int p = 1; p < 3; p++) {
    for (int t = 1; t < o->radix[p]; t *= 2)
      for (int j = 0; j < ns; j++) push((double)j * t, (double)ns * o->radix[p]);
    ns *= o->radix[p];
  }
  MGP_CUDA(cudaMalloc(out, sizeof(float2) * h.size()));
  return upload(c, *out, h.data(), sizeof(float2) * h.size());
}

// Tables of the mesh and, where the lattice transforms apply, of the lattice
// size; the Gaussian smoothing factors exp(-(kR1 d)^2 / 2) per stored index
// (FP64 on the host).  At mgp_create, so that no call allocates or copies
// inside a captured graph.
int mgp_fft_setup(mgp_ctx *c) {
  const int N = c->g.N;
  RET_IF(make_table(c, N, &c->fft_tw));
  if (N % c->Ns == 0 && N != c->Ns) RET_IF(make_table(c, c->Ns, &c->fft_tw_s));
  if (c->p.model == MGP_MODEL_DGP && c->p.smoothing_filter == MGP_FILTER_GAUSSIAN && mgp_fft_has(N)) {
    const double kR1 = (float)(2.0 * M_PI / c->p.Box * c->p.Rsmooth);
    std::vector<float> h(N);
    for (int i = 0; i < N; i++) {
      const double x = kR1 * (i > N / 2 ? i - N : i);
      h[i] = (float)exp(-0.5 * x * x);
    }
    MGP_CUDA(cudaMalloc(&c->fft_gauss, sizeof(float) * N));
    RET_IF(upload(c, c->fft_gauss, h.data(), sizeof(float) * N));
  }
  return MGP_OK;
}

void mgp_fft_free(mgp_ctx *c) {
  float *b[] = {c->fft_tw, c->fft_tw_s, c->fft_gauss, c->fft_scr};
  for (float *p : b)
    if (p) cudaFree(p);
  c->fft_tw = c->fft_tw_s = c->fft_gauss = c->fft_scr = NULL;
}

// ---------------------------------------------------------------- passes
namespace {

// One size's passes over n grids gs floats apart on the context's stream.
struct passes {
  mgp_ctx *c;
  const mgp_fft_ops *o;
  int N, sms;
  const float2 *tw;

  passes(mgp_ctx *ctx, int n) : c(ctx), o(ops_for(n)), N(n), sms(sms_of(ctx)) {
    tw = (const float2 *)(n == ctx->g.N ? ctx->fft_tw : ctx->fft_tw_s);
  }
  bool ok() const { return o && tw; }
  long long rows(int n) const { return (long long)N * N * n; }

  int z(int mode, mgp_fft_z a) const {
    a.tw = tw;
    a.ztw = tw + N;
    return launched(o->z(mode, a, sms, c->stream));
  }
  // n grids, in and out gs floats apart each
  int z_r2c(const float *in, float *out, long long gs, int n) const {
    mgp_fft_z a;
    memset(&a, 0, sizeof(a));
    a.in = (const float2 *)in;
    a.out = (float2 *)out;
    a.rows = rows(n);
    a.bs_in = a.bs_out = gs / 2;
    return z(MGP_Z_R2C, a);
  }
  int z_c2r(const float *in, float *out, long long gs, int n) const { return z_c2r(in, gs, out, gs, n); }
  int z_c2r(const float *in, long long gs_in, float *out, long long gs_out, int n) const {
    mgp_fft_z a;
    memset(&a, 0, sizeof(a));
    a.in = (const float2 *)in;
    a.real = (float2 *)out;
    a.rows = rows(n);
    a.bs_in = gs_in / 2;
    a.bs_real = gs_out / 2;
    return z(MGP_Z_C2R, a);
  }
  // z rows of three spectra to the grids g, g + gs, g + 2 gs: those in the second and
  // third go down by one, the one in `last` to the third, one after the other (a row of
  // a grid and of its spectrum do not lie in the same place).  n boxes.
  int z_c2r_down(float *g, long long gs, long long bs, const float *last, long long bs_last, int n) const {
    RET_IF(z_c2r(g + gs, bs, g, bs, n));
    RET_IF(z_c2r(g + 2 * gs, bs, g + gs, bs, n));
    return z_c2r(last, bs_last, g + 2 * gs, bs, n);
  }
  int y(int dir, float *g, long long gs, int n) const {
    mgp_fft_y a;
    memset(&a, 0, sizeof(a));
    a.ntask = 1;
    a.task[0].in = (const float2 *)g;
    a.task[0].out[0] = (float2 *)g;
    a.task[0].bs_in = a.task[0].bs_out[0] = gs / 2;
    a.task[0].nout = 1;
    return y(dir, 0, a, n);
  }
  int y(int dir, int gen, mgp_fft_y a, int n, int kc = 1 << 30) const {
    a.tw = tw;
    a.nbox = n;
    a.kc = kc;
    return launched(o->y(dir, gen, a, sms, c->stream));
  }
  int x(int fwd, int epi, mgp_fft_x a, int n) const {
    a.tw = tw;
    a.nbox = n;
    return launched(o->x(fwd, epi, a, sms, c->stream));
  }
};

mgp_fft_x x_args(float *in, long long gs) {
  mgp_fft_x a;
  memset(&a, 0, sizeof(a));
  a.in = (const float2 *)in;
  a.spec = (float2 *)in;
  a.bs_in = a.bs_spec = a.bs_o = gs / 2;
  return a;
}

}  // namespace

// Forward transforms of n padded real grids into planar spectra, both gs floats
// apart; in and out do not overlap.
int mgp_fft_r2c(mgp_ctx *c, const float *in, float *out, int n, long long gs) {
  const passes p(c, c->g.N);
  RET_IF(p.z_r2c(in, out, gs, n));
  RET_IF(p.y(-1, out, gs, n));
  return p.x(1, MGP_X_NONE, x_args(out, gs), n);
}

// Inverse transforms of n planar spectra (overwritten) of size N (the mesh or
// the lattice) into padded real grids, both gs floats apart.
int mgp_fft_c2r(mgp_ctx *c, int N, float *in, float *out, int n, long long gs) {
  const passes p(c, N);
  if (!p.ok()) return mgp_set_error(MGP_EINVAL, "no transform of size %d", N);
  mgp_fft_x a = x_args(in, gs);
  a.o[0] = (float2 *)in;
  RET_IF(p.x(0, MGP_X_INV, a, n));
  RET_IF(p.y(1, in, gs, n));
  return p.z_c2r(in, out, gs, n);
}

// The same of the three planar spectra at g + gs, g + 2 gs and last into the grids g,
// g + gs and g + 2 gs.
int mgp_fft_c2r_down(mgp_ctx *c, int N, float *g, float *last, long long gs) {
  const passes p(c, N);
  if (!p.ok()) return mgp_set_error(MGP_EINVAL, "no transform of size %d", N);
  for (int q = 0; q < 2; q++) {
    float *s = q ? last : g + gs;
    const int n = q ? 1 : 2;
    mgp_fft_x a = x_args(s, gs);
    a.o[0] = (float2 *)s;
    RET_IF(p.x(0, MGP_X_INV, a, n));
    RET_IF(p.y(1, s, gs, n));
  }
  return p.z_c2r_down(g, gs, 0, last, 0, 1);
}

// A planar spectrum's x planes x0 .. x1 - 1 in the [N][N][N/2+1] layout.
__global__ void k_planar_rows(const float2 *__restrict__ in, float2 *__restrict__ out, int N, long long rows) {
  const int lane = threadIdx.x & 31, h = N / 2;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
    const long long x = r / N, y = r - x * N;
    const float2 *p = in + x * N * (h + 1);
    float2 *o = out + r * (h + 1);
    for (int k = lane; k < h; k += 32) o[k] = p[y * h + k];
    if (lane == 0) o[h] = p[(long long)N * h + y];
  }
}
int mgp_fft_planar_rows(int N, const float *in, float *out, int x0, int x1, cudaStream_t st) {
  const long long plane = (long long)N * (N / 2 + 1), rows = (long long)(x1 - x0) * N;
  k_planar_rows<<<mgp_blocks_for(rows * 32, 8), 256, 0, st>>>((const float2 *)in + x0 * plane, (float2 *)out, N, rows);
  MGP_CHECK_LAUNCH();
  g_kernel_launches++;
  return MGP_OK;
}

// Scratch spectra of the field passes and the IC: three a box where they are small (256 MB in
// all), so that one launch does the force rows (256^3: 76 us, 88 in three); else a batch takes its density grid, which nothing
// reads after the fifth force's source spectrum, and a single box, which keeps that grid
// for its caller, has one of its own.
int mgp_fft_scratch(mgp_ctx *c) {
  if (c->fft_scr) return MGP_OK;
  const size_t bytes = sizeof(float) * (size_t)c->g.nreal * c->nbox;
  const int grids = 3 * bytes <= (256u << 20) ? 3 : 1;
  if (grids == 1 && c->nbox > 1) return MGP_OK;
  if (cudaMalloc(&c->fft_scr, grids * bytes) != cudaSuccess) {
    cudaGetLastError();
    c->fft_scr = NULL;
    if (c->nbox > 1) return MGP_OK;
    return mgp_set_error(MGP_ECUDA, "no memory for the transforms' scratch grid");
  }
  c->fft_scr_grids = grids;
  return MGP_OK;
}

// The field passes of the PM step (src/auxPM.c:358-555, src/mg.h:21-309) from
// the density in rho: delta(k) in dk, the fifth force's source spectrum in
// rho (both planar), and the three force grids, for all boxes of the context.
// The P(k) and neutrino passes between them are the caller's.  Spectra live in the
// second and third force grid of a box, F1 and F2, and in its scratch grid F3 (three grids
// of scratch a box before, which made the largest batch smaller by a quarter), or in three
// scratch grids:
//   density  rho -> dk; with a filter its inverse x lines -> F1; else, one
//            spectrum being all the forces need, their x lines -> F1, F2
//   screen   F1 -> mg1 (real), rho -> F2
//   force_x  F2 (or dk) -> F1 (k_x G), F2 (G), the source spectrum -> rho
//   force_y  F1 -> F1, F2 -> F2, F3
//   force_z  F1, F2, F3 -> the force grids
static float *frc(const mgp_ctx *c, int q) { return c->frc + (size_t)q * c->g.nreal; }
static bool apart(const mgp_ctx *c) { return c->fft_scr_grids == 3; }
static float *F(const mgp_ctx *c, int q) {
  if (apart(c)) return c->fft_scr + (size_t)(q - 1) * c->g.nreal;
  return q < 3 ? frc(c, q) : (c->nbox == 1 ? c->fft_scr : c->rho);
}
// z rows of F1, F2, F3 to the force grids
static int z_forces(const passes &p) {
  mgp_ctx *c = p.c;
  const long long gs = c->g.nreal;
  if (apart(c)) return p.z_c2r(F(c, 1), c->frc, gs, 3 * c->nbox);
  return p.z_c2r_down(c->frc, gs, 3 * gs, F(c, 3), gs, c->nbox);
}

static mgp_fft_x force_args(mgp_ctx *c, const mgp_fft_plan *f, float *in, long long bs_in, float *spec) {
  mgp_fft_x a = x_args(in, c->g.nreal);
  a.bs_in = bs_in;
  a.spec = (float2 *)spec;
  a.o[0] = (float2 *)F(c, 1);
  a.o[1] = (float2 *)F(c, 2);
  a.bs_o = 3 * c->g.nreal / 2;
  a.mg_kind = f->mg_kind;
  a.cfac = f->cfac;
  a.coupling = f->coupling;
  a.mass2 = f->mass2;
  a.bs = f->bs;
  if (f->mg_kind == 1 || f->mg_kind == 2) {
    a.add = (const float2 *)c->dk;
    a.bs_add = c->g.nreal / 2;
  }
  return a;
}

static mgp_fft_x filter_args(mgp_ctx *c, const mgp_fft_plan *f) {
  mgp_fft_x a = x_args(c->dk, c->g.nreal);
  a.o[0] = (float2 *)F(c, 1);
  a.bs_o = 3 * c->g.nreal / 2;
  a.filter_kind = f->filter_kind;
  a.filter = f->filter;
  a.kR1 = f->kR1;
  a.norm = f->norm;
  a.gauss = c->fft_gauss;
  return a;
}

int mgp_fft_density(mgp_ctx *c, const mgp_fft_plan *f) {
  const passes p(c, c->g.N);
  const int n = c->nbox;
  const long long gs = c->g.nreal;
  RET_IF(mgp_fft_scratch(c));
  RET_IF(p.z_r2c(c->rho, c->dk, gs, n));
  RET_IF(p.y(-1, c->dk, gs, n));
  c->dk_planar = 1;
  if (f->split) return p.x(1, MGP_X_NONE, x_args(c->dk, gs), n);
  if (f->filter_kind) return p.x(1, MGP_X_INV, filter_args(c, f), n);
  if (f->from_rho) return p.x(1, MGP_X_NONE, x_args(c->dk, gs), n);
  return p.x(1, MGP_X_FORCE, force_args(c, f, c->dk, gs / 2, c->dk), n);
}

int mgp_fft_screen(mgp_ctx *c, const mgp_fft_plan *f, int (*user)(mgp_ctx *, const mgp_fft_plan *)) {
  const passes p(c, c->g.N);
  const int n = c->nbox;
  const long long gs = c->g.nreal;
  mgp_fft_z a;
  memset(&a, 0, sizeof(a));
  a.in = (const float2 *)F(c, 1);
  a.out = (float2 *)F(c, 2);
  a.bs_in = a.bs_out = 3 * gs / 2;
  a.real = (float2 *)c->mg1;
  a.rho = (const float2 *)c->rho;
  a.bs_real = gs / 2;
  a.rows = p.rows(n);
  if (f->filter_kind) {
    if (f->split) RET_IF(p.x(0, MGP_X_INV, filter_args(c, f), n));
    RET_IF(p.y(1, F(c, 1), 3 * gs, n));
    if (user) {
      RET_IF(p.z(MGP_Z_C2R, a));
      RET_IF(user(c, f));
    } else {
      a.density = f->filter_kind == 1;
      a.phicrit = f->phicrit;
      a.coupling = f->screen_coupling;
      a.pref = f->screen_pref;
      a.base = f->screen_base;
      a.scalars = f->bs;
      RET_IF(p.z(MGP_Z_SCREEN, a));
    }
  }
  if (!f->filter_kind || user) {
    a.in = (const float2 *)c->rho;
    a.bs_in = gs / 2;
    RET_IF(p.z(MGP_Z_R2C, a));
  }
  return p.y(-1, F(c, 2), 3 * gs, n);
}

int mgp_fft_force_x(mgp_ctx *c, const mgp_fft_plan *f) {
  const passes p(c, c->g.N);
  const long long gs = c->g.nreal;
  if (!f->from_rho) return p.x(0, MGP_X_FORCE, force_args(c, f, c->dk, gs / 2, NULL), c->nbox);
  RET_IF(p.x(1, MGP_X_FORCE, force_args(c, f, F(c, 2), 3 * gs / 2, c->rho), c->nbox));
  c->rho_planar = 1;
  return MGP_OK;
}

// y pass of the force fields kx G in F1 and G in F2 after their x lines: F_x in F1, F_y =
// ky G in F2, F_z = kz G in F3
static mgp_fft_y force_y_args(const mgp_ctx *c) {
  const long long bs = 3 * c->g.nreal / 2;
  mgp_fft_y a;
  memset(&a, 0, sizeof(a));
  a.ntask = 2;
  a.task[0].in = a.task[0].out[0] = (float2 *)F(c, 1);
  a.task[0].bs_in = a.task[0].bs_out[0] = bs;
  a.task[0].nout = 1;
  a.task[1].in = a.task[1].out[0] = (float2 *)F(c, 2);
  a.task[1].bs_in = a.task[1].bs_out[0] = bs;
  a.task[1].ypow[0] = 1;
  a.task[1].out[1] = (float2 *)F(c, 3);
  a.task[1].bs_out[1] = apart(c) ? bs : c->g.nreal / 2;
  a.task[1].zpow[1] = 1;
  a.task[1].nout = 2;
  return a;
}

int mgp_fft_force_y(mgp_ctx *c) { return passes(c, c->g.N).y(1, 1, force_y_args(c), c->nbox); }

int mgp_fft_force_z(mgp_ctx *c) { return z_forces(passes(c, c->g.N)); }

// The 2LPT source's spectrum in rho from delta(k) in dk (src/2LPT.c:1224-1290),
// both planar, for all boxes: three inverse x transforms of -delta / k^2 times 1,
// kx, kx^2, from them six y transforms of the gradients, then one row pass that
// inverts the six rows, forms the source and transforms it forward.  delta is
// zero beyond |k| <= kc: columns and tiles beyond it are skipped (at Nmesh = 2
// Nsample a quarter of the x columns and half of the y columns are left).
// A box's six gradients take the force grids: of two boxes in a batch, which goes by as
// many boxes as have room there; a single box has its scratch and, with one grid of it,
// two more.
int mgp_fft_ic_source(mgp_ctx *c, int kc) {
  const passes p(c, c->g.N);
  const long long gs = c->g.nreal;
  const int per = c->nbox == 1 ? 1 : c->nbox / 2;
  RET_IF(mgp_fft_scratch(c));
  const int own = c->nbox > 1 ? 3 : c->fft_scr_grids;
  if (own == 1) RET_IF(mgp_ic_scratch(c, 2));
  float2 *g[6];
  for (int q = 0; q < 6; q++) {
    float *more = c->nbox > 1 ? frc(c, 3) : c->fft_scr;
    g[q] = (float2 *)(q < 3 ? frc(c, q) : q < 3 + own ? more + (q - 3) * gs : c->ic_scratch + (q - 4) * gs);
  }
  for (int b = 0; b < c->nbox; b += per) {
    const int n = c->nbox - b < per ? c->nbox - b : per;
    mgp_fft_x x = x_args(c->dk + b * gs, gs);
    x.o[0] = g[5];
    x.o[1] = g[2];
    x.o[2] = g[0];
    x.bs_o = 6 * gs / 2;
    x.kc = kc;
    RET_IF(p.x(0, MGP_X_IC, x, n));
    mgp_fft_y y;
    memset(&y, 0, sizeof(y));
    y.ntask = 3;
    y.neg = 1;
    y.task[0].in = y.task[0].out[0] = g[0];
    y.task[0].nout = 1;
    y.task[1].in = g[2];
    y.task[1].out[0] = g[1];
    y.task[1].ypow[0] = 1;
    y.task[1].out[1] = g[2];
    y.task[1].zpow[1] = 1;
    y.task[1].nout = 2;
    y.task[2].in = g[5];
    y.task[2].out[0] = g[3];
    y.task[2].ypow[0] = 2;
    y.task[2].out[1] = g[4];
    y.task[2].ypow[1] = y.task[2].zpow[1] = 1;
    y.task[2].out[2] = g[5];
    y.task[2].zpow[2] = 2;
    y.task[2].nout = 3;
    for (int t = 0; t < 3; t++) {
      y.task[t].bs_in = 6 * gs / 2;
      for (int q = 0; q < 3; q++) y.task[t].bs_out[q] = 6 * gs / 2;
    }
    RET_IF(p.y(1, 1, y, n, kc));
    mgp_fft_z z;
    memset(&z, 0, sizeof(z));
    for (int q = 0; q < 6; q++) z.grad[q] = g[q];
    z.out = (float2 *)(c->rho + b * gs);
    z.rows = p.rows(n);
    z.bs_in = 6 * gs / 2;
    z.bs_out = gs / 2;
    z.kc = kc;
    RET_IF(p.z(MGP_Z_SOURCE, z));
  }
  RET_IF(p.y(-1, c->rho, gs, c->nbox));
  c->rho_planar = 1;
  return p.x(1, MGP_X_NONE, x_args(c->rho, gs), c->nbox);
}

// The particles' D1, D2, s and v from delta(k) in dk and the 2LPT source in rho.
int mgp_fft_ic_fields(mgp_ctx *c) {
  const int N = c->g.N, Ns = c->Ns, n = c->nbox;
  const long long gs = c->g.nreal;
  const float mult = (float)(-3.0 / 7.0 / ((double)N * N * N));
  // D1: three cuFFT transforms in the force grids
  RET_IF(mgp_launch_ic_za(c->dk, c->frc, gs, N, c->p.Box, n, c->stream));
  for (int g = 0; g < 3; g++)
    MGP_CUFFT(cufftExecC2R(n > 1 ? c->plan_c2r_frc_b : c->plan_c2r_1, (cufftComplex *)(c->frc + g * gs),
                           (cufftReal *)(c->frc + g * gs)));
  RET_IF(mgp_launch_ic_take(c->frc, 3 * gs, gs, N, N / Ns, Ns, c->np, c->ic_box, n, 0, 1.0f, c->D1, c->D2, c->s, c->v,
                            c->stream));
  if (N != Ns) {
    // three lattice grids a box, all boxes' spectra and then all grids in the force
    // grids (at most 3/4 of a mesh grid a box)
    const long long ls = (long long)Ns * Ns * (Ns + 2);
    float *out = c->frc + 3 * n * ls;
    RET_IF(mgp_launch_ic_fold(c->rho, gs, N, Ns, c->p.Box, c->frc, ls, n, c->stream));
    RET_IF(mgp_fft_c2r(c, Ns, c->frc, out, 3 * n, ls));
    return mgp_launch_ic_take(out, 3 * ls, ls, Ns, 1, Ns, c->np, c->ic_box, n, 1, mult, c->D1, c->D2, c->s, c->v,
                              c->stream);
  }
  // the force pass's x, y and z passes with g = -Box/2pi / k^2 on the source
  const passes p(c, N);
  mgp_fft_x x = x_args(c->rho, gs);
  x.o[0] = (float2 *)F(c, 1);
  x.o[1] = (float2 *)F(c, 2);
  x.bs_o = 3 * gs / 2;
  x.cfac = (float)(-c->p.Box / (2.0 * M_PI));
  x.neg = 1;
  RET_IF(p.x(0, MGP_X_FORCE, x, n));
  mgp_fft_y y = force_y_args(c);
  y.neg = 1;
  RET_IF(p.y(1, 1, y, n));
  RET_IF(z_forces(p));
  return mgp_launch_ic_take(c->frc, 3 * gs, gs, N, 1, Ns, c->np, c->ic_box, n, 1, mult, c->D1, c->D2, c->s, c->v,
                            c->stream);
}
