// hmcops.cu -- the gauge and momentum side of an HMC step on the device:
//  - gauge action (gaugeAction1, src/gauge/gaugeAction.nim:487-571) and
//    gauge force (gaugeForce = gaugeActionDeriv + contractProjectTAH,
//    gaugeAction.nim:576-779, src/gauge/gaugeUtils.nim:419-441) for
//    plaquette + rectangle (Symanzik / Iwasaki / DBW2) coefficients;
//  - link update U <- expAH(eps P) U (axexpmuly, gaugeUtils.nim:452-459;
//    expAH, src/maths/matexp.nim:316-346);
//  - momentum update P += a F and refresh P = randomTAH (randTah3,
//    gaugeUtils.nim:1466-1493) from a counter-based generator;
//  - kinetic energy 0.5 |P|^2 - 16 V (kineticAction,
//    src/hmc/hmcAction.nim:248-255).
// Fields are 4-direction link fields double2[4][9][V] (the library's link
// layout).  The force gathers, per (site, direction), every plaquette and
// 2x1 rectangle through the link, with the block order of the smearing sweeps.
#include <algorithm>

#include "smear.cuh"

namespace qs {

// t = t (F or F^dag) at site s; F streamed a row (or column) at a time
__device__ __forceinline__ void mul_link(M3 &t, const double2 *F, size_t V, int s, bool dag) {
  M3 r;
#pragma unroll
  for (int e = 0; e < 9; e++) r.e[e] = make_double2(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 f[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      // (F^dag)_kj = conj(F_jk)
      const double2 v = __ldg(F + (size_t)(dag ? 3 * j + k : 3 * k + j) * V + s);
      f[j] = dag ? make_double2(v.x, -v.y) : v;
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) r.e[3 * i + j] = cmadd(r.e[3 * i + j], t.e[3 * i + k], f[j]);
  }
  t = r;
}
__device__ __forceinline__ void set_link(M3 &t, const double2 *F, size_t V, int s, bool dag) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 v = __ldg(F + (size_t)(dag ? 3 * j + i : 3 * i + j) * V + s);
      t.e[3 * i + j] = dag ? make_double2(v.x, -v.y) : v;
    }
}

struct PathCtx {
  const Geom *g;
  const SiteCtx *c;
  const double2 *u;
  int mu, nu;
};
// site x + a mu + b nu
__device__ __forceinline__ int at(const PathCtx &p, int a, int b) {
  if (b == 0) return a == 0 ? p.c->site : disp1(*p.g, p.c->x, p.c->lex, p.c->par, p.mu, a);
  if (a == 0) return disp1(*p.g, p.c->x, p.c->lex, p.c->par, p.nu, b);
  return disp2(*p.g, p.c->x, p.c->lex, p.c->par, p.mu, a, p.nu, b);
}
// one step of an open path: along +-nu from (a, b), or -mu from (a, b)
__device__ __forceinline__ void step_nu(M3 &t, const PathCtx &p, int a, int b, int s, bool first) {
  const size_t V = (size_t)p.g->V;
  const double2 *Un = p.u + (size_t)p.nu * 9 * V;
  const int site = s > 0 ? at(p, a, b) : at(p, a, b - 1);
  if (first)
    set_link(t, Un, V, site, s < 0);
  else
    mul_link(t, Un, V, site, s < 0);
}
__device__ __forceinline__ void step_back_mu(M3 &t, const PathCtx &p, int a, int b) {
  const size_t V = (size_t)p.g->V;
  mul_link(t, p.u + (size_t)p.mu * 9 * V, V, at(p, a - 1, b), true);
}

// acc += cp * (plaquette closers) + cr * (rectangle closers) of U_mu(x):
// open paths from x+mu back to x (Re Tr[U_mu(x) C] is the loop)
__device__ __forceinline__ void closers(M3 &acc, const Geom &g, const SiteCtx &c, const double2 *u, int mu,
                                        double cp, double cr) {
  const size_t V = (size_t)g.V;
#pragma unroll 1
  for (int k = 0; k < 3; k++) {
    PathCtx p{&g, &c, u, mu, other_dir(mu, k)};
#pragma unroll 1
    for (int s = -1; s <= 1; s += 2) {
      M3 t;
      // plaquette: x+mu -> x+mu+s nu -> x+s nu -> x
      step_nu(t, p, 1, 0, s, true);
      step_back_mu(t, p, 1, s);
      step_nu(t, p, 0, s, -s, false);
      m_axpy(acc, cp, t);
      if (cr == 0.0) continue;
      // long in mu, U_mu(x) first: x+mu -> x+2mu -> +s nu -> back 2 mu -> x
      set_link(t, u + (size_t)mu * 9 * V, V, at(p, 1, 0), false);
      step_nu(t, p, 2, 0, s, false);
      step_back_mu(t, p, 2, s);
      step_back_mu(t, p, 1, s);
      step_nu(t, p, 0, s, -s, false);
      m_axpy(acc, cr, t);
      // long in mu, U_mu(x) second: x+mu -> +s nu -> back 2 mu -> x-mu -> x
      step_nu(t, p, 1, 0, s, true);
      step_back_mu(t, p, 1, s);
      step_back_mu(t, p, 0, s);
      step_nu(t, p, -1, s, -s, false);
      mul_link(t, u + (size_t)mu * 9 * V, V, at(p, -1, 0), false);
      m_axpy(acc, cr, t);
      // long in nu: x+mu -> x+mu+2s nu -> x+2s nu -> x
      step_nu(t, p, 1, 0, s, true);
      step_nu(t, p, 1, s, s, false);
      step_back_mu(t, p, 1, 2 * s);
      step_nu(t, p, 0, 2 * s, -s, false);
      step_nu(t, p, 0, s, -s, false);
      m_axpy(acc, cr, t);
    }
  }
}

__device__ __forceinline__ void tah(M3 &r, const M3 &m) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 a = m.e[3 * i + j], b = m.e[3 * j + i];
      r.e[3 * i + j] = make_double2(0.5 * (a.x - b.x), 0.5 * (a.y + b.y));
    }
  const double t = (r.e[0].y + r.e[4].y + r.e[8].y) * (1.0 / 3.0);
  r.e[0].y -= t;
  r.e[4].y -= t;
  r.e[8].y -= t;
}

// F_mu(x) = projectTAH(U_mu(x) (cp sum P + cr sum R)), cp = plaq/3, cr = rect/3,
// path by path: without rectangles (two products per path, nothing to share),
// and where the scratch of the two-sweep form below cannot be had
__global__ void __launch_bounds__(kSmBlock) gauge_force_kernel(Geom g, const double2 *__restrict__ u, double2 *f,
                                                               double cp, double cr) {
  SiteCtx c;
  if (!site_of_thread(g, c)) return;
  const int mu = c.mu;
  const size_t V = (size_t)g.V;
  M3 acc;
#pragma unroll
  for (int e = 0; e < 9; e++) acc.e[e] = make_double2(0.0, 0.0);
  closers(acc, g, c, u, mu, cp, cr);
  M3 um, m, r;
  m_load(um, u + (size_t)mu * 9 * V, V, c.site);
  m_nn(m, um, acc);
  tah(r, m);
  m_store(f + (size_t)mu * 9 * V, V, c.site, r);
}

// ---------------------------------------------------------------------------
// The force in two sweeps.  With A_mu(x) the weighted sum of the open paths
// beside U_mu(x), F_mu = projectTAH(U_mu A_mu^dag).  Every 2x1 rectangle is a
// plaquette one of whose links is replaced by its own staple, so a first
// sweep stores the two halves of every staple,
//   Up_{mu,nu}(x) = U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag
//   Dn_{mu,nu}(x) = U_nu(x)^dag U_mu(x) U_nu(x+mu)      (a path beside U_mu(x+nu))
// and the second adds, with W = U_mu(x+nu), V = U_nu(x+mu) above the link and
// z = x-nu, W = U_mu(z), V = U_nu(z+mu) below it,
//   U_nu(x) [cp W V^dag + cr Up_{mu,nu}(x+nu) V^dag + cr W Up_{nu,mu}(x+mu)^dag]
//     + cr Dn_{nu,mu}(x-mu) W V^dag
//   U_nu(z)^dag [cp W V + cr Dn_{mu,nu}(z-nu) V + cr W Up_{nu,mu}(z+mu)]
//     + cr Dn_{nu,mu}(z-mu)^dag W V.
// 42 3x3 products per link where following each path took 84.  The
// sweeps go through the lattice in slabs of time slices, with two slices
// below and one above of their own, so that the 24 fields of 144 B per site
// take at most kGaugeScratch (any lattice up to 32^4 is one slab).
//
// Bound by what L2 delivers (36 matrices a link) and FP64 issue.  24^4: 255 us
// for the halves and 651 us for the force (255 registers and 8 warps an SM; 758
// us at 168 registers, which spill), against 1670 us path by path.
// ---------------------------------------------------------------------------

struct GaugeArgs {
  Geom g;
  const double2 *u;
  double2 *f;
  double2 *up, *dn;  // [4][3][9][2 nk]: parity blocks of the slab's nk half sites
  int k0, nk;        // the slab: half sites k0 .. k0 + nk - 1, periodic
  int o0, on;        // the half sites whose force this launch forms
  double cp, cr;
};

// Block b works on direction b % 4 and both parities of 64 half sites
// (start .. start + n - 1, periodic) of the list.
__device__ __forceinline__ bool site_of_slab(const Geom &g, SiteCtx &c, int start, int n) {
  const int b = blockIdx.x, w = threadIdx.x >> 5;
  c.mu = b & 3;
  c.par = w & 1;
  const int i = (b >> 2) * (kSmBlock / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  if (i >= n) return false;
  int k = start + i;
  if (k >= g.nh) k -= g.nh;
  c.site = c.par * g.nh + k;
  site_coords(g, c.par, k, c.x, c.lex);
  return true;
}
inline int slab_grid(int n) { return 4 * ((n + kSmBlock / 2 - 1) / (kSmBlock / 2)); }

// place of a site in the slab's fields
__device__ __forceinline__ int in_slab(const GaugeArgs &A, int site) {
  const int par = site >= A.g.nh ? 1 : 0;
  int d = site - par * A.g.nh - A.k0;
  if (d < 0) d += A.g.nh;
  return par * A.nk + d;
}

__device__ __forceinline__ void ld_row(double2 r[3], const double2 *__restrict__ F, size_t V, int s, int i) {
#pragma unroll
  for (int k = 0; k < 3; k++) r[k] = __ldg(F + (size_t)(3 * i + k) * V + s);
}
__device__ __forceinline__ void ld_col(double2 r[3], const double2 *__restrict__ F, size_t V, int s, int k) {
#pragma unroll
  for (int i = 0; i < 3; i++) r[i] = __ldg(F + (size_t)(3 * i + k) * V + s);
}
// out_j += (row r) m or (row r) m^dag
__device__ __forceinline__ void row_nn(double2 *out, const double2 r[3], const M3 &m) {
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int k = 0; k < 3; k++) out[j] = cmadd(out[j], r[k], m.e[3 * k + j]);
}
__device__ __forceinline__ void row_nd(double2 *out, const double2 r[3], const M3 &m) {
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int k = 0; k < 3; k++) out[j] = cjmadd(out[j], m.e[3 * j + k], r[k]);
}
__device__ __forceinline__ void scale3(double2 r[3], double a) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    r[k].x *= a;
    r[k].y *= a;
  }
}
// acc += (column c of a matrix) (row r), or with conj(c)
__device__ __forceinline__ void outer_nn(M3 &acc, const double2 c[3], const double2 *r) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) acc.e[3 * i + j] = cmadd(acc.e[3 * i + j], c[i], r[j]);
}
__device__ __forceinline__ void outer_dn(M3 &acc, const double2 c[3], const double2 *r) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) acc.e[3 * i + j] = cjmadd(acc.e[3 * i + j], c[i], r[j]);
}

__global__ void __launch_bounds__(kSmBlock, 3) gauge_halves_kernel(const GaugeArgs A) {
  SiteCtx c;
  const Geom &g = A.g;
  if (!site_of_slab(g, c, A.k0, A.nk)) return;
  const int mu = c.mu;
  const size_t V = (size_t)g.V, N = (size_t)2 * A.nk;
  const int here = in_slab(A, c.site);
  const double2 *Um = A.u + (size_t)mu * 9 * V;
  const int s_pm = disp1(g, c.x, c.lex, c.par, mu, 1);
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    const int nu = other_dir(mu, j);
    const double2 *Un = A.u + (size_t)nu * 9 * V;
    const int s_pn = disp1(g, c.x, c.lex, c.par, nu, 1);
    double2 *up = A.up + (size_t)(mu * 3 + j) * 9 * N + here, *dn = A.dn + (size_t)(mu * 3 + j) * 9 * N + here;
    M3 v, t;
    m_load(v, Un, V, s_pm);
    m_zero(t);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double2 r[3];
      ld_row(r, Um, V, s_pn, i);
      row_nd(t.e + 3 * i, r, v);  // U_mu(x+nu) V^dag
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double2 r[3], o[3] = {};
      ld_row(r, Un, V, c.site, i);
      row_nn(o, r, t);
#pragma unroll
      for (int k = 0; k < 3; k++) up[(size_t)(3 * i + k) * N] = o[k];
    }
    m_zero(t);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double2 r[3];
      ld_row(r, Um, V, c.site, i);
      row_nn(t.e + 3 * i, r, v);  // U_mu(x) V
    }
    m_zero(v);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double2 r[3];
      ld_row(r, Un, V, c.site, k);
      outer_dn(v, r, t.e + 3 * k);
    }
#pragma unroll
    for (int e = 0; e < 9; e++) dn[(size_t)e * N] = v.e[e];
  }
}

__global__ void __launch_bounds__(kSmBlock, 2) gauge_rect_force_kernel(const GaugeArgs A) {
  SiteCtx c;
  const Geom &g = A.g;
  if (!site_of_slab(g, c, A.o0, A.on)) return;
  const int mu = c.mu;
  const size_t V = (size_t)g.V, N = (size_t)2 * A.nk;
  const double2 *Um = A.u + (size_t)mu * 9 * V;
  const double cp = A.cp, cr = A.cr;
  M3 acc;
  m_zero(acc);
  const int s_pm = disp1(g, c.x, c.lex, c.par, mu, 1);
  const int l_pm = in_slab(A, s_pm), l_mm = in_slab(A, disp1(g, c.x, c.lex, c.par, mu, -1));
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    const int nu = other_dir(mu, j);
    const double2 *Un = A.u + (size_t)nu * 9 * V;
    const double2 *up_mn = A.up + (size_t)(mu * 3 + j) * 9 * N, *dn_mn = A.dn + (size_t)(mu * 3 + j) * 9 * N;
    const int jm = nu * 3 + other_index(nu, mu);
    const double2 *up_nm = A.up + (size_t)jm * 9 * N, *dn_nm = A.dn + (size_t)jm * 9 * N;
    M3 v, P, K;
    // above the link
    {
      const int s_pn = disp1(g, c.x, c.lex, c.par, nu, 1);
      const int l_pn = in_slab(A, s_pn);
      m_load(v, Un, V, s_pm);
      m_zero(P);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 r[3];
        ld_row(r, Um, V, s_pn, i);
        row_nd(P.e + 3 * i, r, v);
#pragma unroll
        for (int k = 0; k < 3; k++) K.e[3 * i + k] = make_double2(cp * P.e[3 * i + k].x, cp * P.e[3 * i + k].y);
        ld_row(r, up_mn, N, l_pn, i);
        scale3(r, cr);
        row_nd(K.e + 3 * i, r, v);
      }
      m_load(v, up_nm, N, l_pm);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 r[3];
        ld_row(r, Um, V, s_pn, i);
        scale3(r, cr);
        row_nd(K.e + 3 * i, r, v);
      }
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double2 r[3];
        ld_col(r, Un, V, c.site, k);
        outer_nn(acc, r, K.e + 3 * k);
        ld_col(r, dn_nm, N, l_mm, k);
        scale3(r, cr);
        outer_nn(acc, r, P.e + 3 * k);
      }
    }
    // below it
    {
      const int z = disp1(g, c.x, c.lex, c.par, nu, -1), zpm = disp2(g, c.x, c.lex, c.par, nu, -1, mu, 1);
      const int l_2 = in_slab(A, disp1(g, c.x, c.lex, c.par, nu, -2));
      const int l_zpm = in_slab(A, zpm), l_zmm = in_slab(A, disp2(g, c.x, c.lex, c.par, nu, -1, mu, -1));
      m_load(v, Un, V, zpm);
      m_zero(P);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 r[3];
        ld_row(r, Um, V, z, i);
        row_nn(P.e + 3 * i, r, v);
#pragma unroll
        for (int k = 0; k < 3; k++) K.e[3 * i + k] = make_double2(cp * P.e[3 * i + k].x, cp * P.e[3 * i + k].y);
        ld_row(r, dn_mn, N, l_2, i);
        scale3(r, cr);
        row_nn(K.e + 3 * i, r, v);
      }
      m_load(v, up_nm, N, l_zpm);
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 r[3];
        ld_row(r, Um, V, z, i);
        scale3(r, cr);
        row_nn(K.e + 3 * i, r, v);
      }
#pragma unroll
      for (int k = 0; k < 3; k++) {
        double2 r[3];
        ld_row(r, Un, V, z, k);
        outer_dn(acc, r, K.e + 3 * k);
        ld_row(r, dn_nm, N, l_zmm, k);
        scale3(r, cr);
        outer_dn(acc, r, P.e + 3 * k);
      }
    }
  }
  M3 um, m;
  m_load(um, Um, V, c.site);
  m_nd(m, um, acc);
  tah(um, m);
  m_store(A.f + (size_t)mu * 9 * V, V, c.site, um);
}

constexpr size_t kGaugeScratch = (size_t)4 << 30;

// the plaquette and rectangle force through the slabs; QEXSTAG_ERR_ALLOC (with
// nothing launched) where their scratch cannot be had
static int rect_force_dev(qexstag_layout_s *l, const double2 *u, double2 *f, double cp, double cr) {
  const Geom &g = l->g;
  const int T = g.L[3], sh = g.nh / T;  // half sites of a time slice
  const size_t slice = (size_t)24 * 9 * sizeof(double2) * 2 * sh;
  // slices of force per slab, and of scratch
  int n = T, held = T;
  if (slice * T > kGaugeScratch) {
    held = (int)(kGaugeScratch / slice);  // < T
    n = held - 3;
    if (n < 1) return QEXSTAG_ERR_ALLOC;
  }
  void *p = l->scratch.take(slice * held);
  if (!p) return QEXSTAG_ERR_ALLOC;
  GaugeArgs A;
  A.g = g;
  A.u = u;
  A.f = f;
  A.nk = held * sh;
  A.up = (double2 *)p;
  A.dn = A.up + (size_t)12 * 9 * 2 * A.nk;
  A.cp = cp;
  A.cr = cr;
  for (int t = 0; t < T; t += n) {
    const int here = std::min(n, T - t);
    A.k0 = held == T ? 0 : ((t - 2 + T) % T) * sh;
    A.o0 = t * sh;
    A.on = here * sh;
    gauge_halves_kernel<<<slab_grid(A.nk), kSmBlock, 0, stream()>>>(A);
    gauge_rect_force_kernel<<<slab_grid(A.on), kSmBlock, 0, stream()>>>(A);
    note_launch(2);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
  l->scratch.give(p);
  return e == cudaSuccess ? QEXSTAG_OK : cuda_fail(e, "gauge_force");
}

// sum_{x, mu>nu} Re Tr P and sum_{x, mu!=nu} Re Tr R (long side mu), each
// loop once, as Re Tr[U_mu(x) C] over the loops' first links.  With the one block
// on an SM that 244 registers leave, the next link's loads are on their way while
// a product is formed: 24^4 with rectangles 364 us without the bound (170
// registers, the same one block), 314; two blocks (128, with spills) 339.
__global__ void __launch_bounds__(kBlock, 1) gauge_action_kernel(Geom g, const double2 *__restrict__ u, int rect,
                                                              double *partials, unsigned *ticket, double *out) {
  double s[2] = {0.0, 0.0};
  const size_t V = (size_t)g.V;
  for (int site = blockIdx.x * blockDim.x + threadIdx.x; site < g.V; site += gridDim.x * blockDim.x) {
    SiteCtx c;
    c.site = site;
    c.par = site >= g.nh ? 1 : 0;
    site_coords(g, c.par, site - c.par * g.nh, c.x, c.lex);
#pragma unroll 1
    for (int mu = 0; mu < 4; mu++) {
      c.mu = mu;
#pragma unroll 1
      for (int nu = 0; nu < 4; nu++) {
        if (nu == mu) continue;
        PathCtx p{&g, &c, u, mu, nu};
        M3 t, um, m;
        m_load(um, u + (size_t)mu * 9 * V, V, site);
        if (nu < mu) {
          step_nu(t, p, 1, 0, 1, true);
          step_back_mu(t, p, 1, 1);
          step_nu(t, p, 0, 1, -1, false);
          m_nn(m, um, t);
          s[0] += m.e[0].x + m.e[4].x + m.e[8].x;
        }
        if (rect) {
          set_link(t, u + (size_t)mu * 9 * V, V, at(p, 1, 0), false);
          step_nu(t, p, 2, 0, 1, false);
          step_back_mu(t, p, 2, 1);
          step_back_mu(t, p, 1, 1);
          step_nu(t, p, 0, 1, -1, false);
          m_nn(m, um, t);
          s[1] += m.e[0].x + m.e[4].x + m.e[8].x;
        }
      }
    }
  }
  double tot[2];
  if (grid_reduce<2>(s, partials, ticket, tot) && threadIdx.x == 0) {
    out[0] = tot[0];
    out[1] = tot[1];
  }
}

// expAH(x): scale until |x|^2 <= 1/16, degree-12 Taylor polynomial in
// Paterson-Stockmeyer form (x, x^2, x^3), square back (matexp.nim:316-346)
__device__ __forceinline__ void exp_ah(M3 &r, const M3 &x0) {
  double n2 = 0.0;
#pragma unroll
  for (int e = 0; e < 9; e++) n2 += x0.e[e].x * x0.e[e].x + x0.e[e].y * x0.e[e].y;
  double scale = 1.0;
  int ns = 0;
  while (n2 > 1.0 / 16.0 && ns < 64) {
    n2 *= 0.25;
    scale *= 0.5;
    ns++;
  }
  M3 m = x0, m2, m3, a;
  m_scale(m, scale);
  m_nn(m2, m, m);
  m_nn(m3, m2, m);
  const double c2 = 0.5, c3 = 1.0 / 6, c4 = 1.0 / 24, c5 = 1.0 / 120, c6 = 1.0 / 720, c7 = 1.0 / 5040,
               c8 = 1.0 / 40320, c9 = 1.0 / 362880, c10 = 1.0 / 3628800, c11 = 1.0 / 39916800,
               c12 = 1.0 / 479001600;
  // a = c12 m3 + c11 m2 + c10 m + c9
#pragma unroll
  for (int e = 0; e < 9; e++)
    a.e[e] = make_double2(c12 * m3.e[e].x + c11 * m2.e[e].x + c10 * m.e[e].x,
                          c12 * m3.e[e].y + c11 * m2.e[e].y + c10 * m.e[e].y);
  a.e[0].x += c9;
  a.e[4].x += c9;
  a.e[8].x += c9;
  // a <- a m3 + c8 m2 + c7 m + c6, then + c5 m2 + c4 m + c3, then + c2 m2 + m + 1
  const double k2[3] = {c8, c5, c2}, k1[3] = {c7, c4, 1.0}, k0[3] = {c6, c3, 1.0};
#pragma unroll 1
  for (int s = 0; s < 3; s++) {
    m_nn(r, a, m3);
#pragma unroll
    for (int e = 0; e < 9; e++) {
      r.e[e].x += k2[s] * m2.e[e].x + k1[s] * m.e[e].x;
      r.e[e].y += k2[s] * m2.e[e].y + k1[s] * m.e[e].y;
    }
    r.e[0].x += k0[s];
    r.e[4].x += k0[s];
    r.e[8].x += k0[s];
    a = r;
  }
#pragma unroll 1
  for (int k = 0; k < ns; k++) {
    m_nn(r, a, a);
    a = r;
  }
  r = a;
}

__global__ void __launch_bounds__(kSmBlock) link_update_kernel(int V, double2 *u, const double2 *__restrict__ p,
                                                               double eps) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const size_t off = (size_t)blockIdx.y * 9 * V;
  M3 x, e, y, z;
  m_load(x, p + off, (size_t)V, s);
  m_scale(x, eps);
  exp_ah(e, x);
  m_load_own(y, u + off, (size_t)V, s);
  m_nn(z, e, y);
  m_store(u + off, (size_t)V, s, z);
}

__global__ void axpy_field_kernel(size_t n, double2 *y, double a, const double2 *__restrict__ x) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = x[i];
    double2 w = y[i];
    w.x = fma(a, v.x, w.x);
    w.y = fma(a, v.y, w.y);
    y[i] = w;
  }
}

// ---- Philox-4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) ----
__device__ __forceinline__ uint4 philox4x32(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}
// uniform in (0, 1) from 64 random bits (53 used)
__device__ __forceinline__ double unit_open(uint32_t a, uint32_t b) {
  const uint64_t v = ((uint64_t)a << 21) ^ (uint64_t)(b >> 11);  // 53 bits
  return ((double)(v & ((1ull << 53) - 1)) + 0.5) * (1.0 / 9007199254740992.0);
}

// P = randTah3 per link (gaugeUtils.nim:1466-1493): Gaussian coefficients
// with the sqrt(1/2), sqrt(1/3) normalisation; link k of the field draws
// from counter (k, counter), key seed
__global__ void momenta_heatbath_kernel(int V, double2 *p, uint2 key, uint32_t clo, uint32_t chi) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const int mu = blockIdx.y;
  const uint32_t link = (uint32_t)mu * (uint32_t)V + (uint32_t)s;
  double gs[8];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const uint4 r0 = philox4x32(make_uint4(link, clo, chi, 2u * q), key);
    const uint4 r1 = philox4x32(make_uint4(link, clo, chi, 2u * q + 1u), key);
    const double u1 = unit_open(r0.x, r0.y), u2 = unit_open(r0.z, r0.w);
    const double u3 = unit_open(r1.x, r1.y), u4 = unit_open(r1.z, r1.w);
    const double ra = sqrt(-2.0 * log(u1)), rb = sqrt(-2.0 * log(u3));
    double sa, ca, sb, cb;
    sincospi(2.0 * u2, &sa, &ca);
    sincospi(2.0 * u4, &sb, &cb);
    gs[4 * q + 0] = ra * ca;
    gs[4 * q + 1] = ra * sa;
    gs[4 * q + 2] = rb * cb;
    gs[4 * q + 3] = rb * sb;
  }
  const double s2 = 0.70710678118654752440, s3 = 0.57735026918962576450;
  const double r3 = s2 * gs[0], r8 = s2 * s3 * gs[1];
  const double r01 = s2 * gs[2], r02 = s2 * gs[3], r12 = s2 * gs[4];
  const double i01 = s2 * gs[5], i02 = s2 * gs[6], i12 = s2 * gs[7];
  M3 m;
  m.e[0] = make_double2(0.0, r8 + r3);
  m.e[4] = make_double2(0.0, r8 - r3);
  m.e[8] = make_double2(0.0, -2.0 * r8);
  m.e[1] = make_double2(r01, i01);
  m.e[3] = make_double2(-r01, i01);
  m.e[2] = make_double2(r02, i02);
  m.e[6] = make_double2(-r02, i02);
  m.e[5] = make_double2(r12, i12);
  m.e[7] = make_double2(-r12, i12);
  m_store(p + (size_t)mu * 9 * V, (size_t)V, s, m);
}

__global__ void __launch_bounds__(kBlock) norm2_field_kernel(size_t n, const double2 *__restrict__ x, double *partials,
                                                             unsigned *ticket, double *out) {
  double s[1] = {0.0};
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = x[i];
    s[0] += v.x * v.x + v.y * v.y;
  }
  double tot[1];
  if (grid_reduce<1>(s, partials, ticket, tot) && threadIdx.x == 0) out[0] = tot[0];
}

// a 4-direction link field given in either memory space, staged on the
// device for host callers
struct Field4 {
  const Geom *g = nullptr;
  double2 *dev = nullptr;
  void *own = nullptr;
  double *host = nullptr;
  ~Field4() {
    if (own) {
      cudaStreamSynchronize(stream());
      cudaFree(own);
    }
  }
};

static int field_in(const Geom &g, const double *p, int mem, bool upload, Field4 &f) {
  f.g = &g;
  if (mem == QEXSTAG_MEM_DEVICE) {
    f.dev = (double2 *)p;
    return QEXSTAG_OK;
  }
  const size_t per = sizeof(double2) * 9 * (size_t)g.V;
  if (device_malloc(&f.own, 5 * per) != cudaSuccess) {
    cudaGetLastError();
    return fail(QEXSTAG_ERR_ALLOC, "device allocation failed");
  }
  f.dev = (double2 *)f.own;
  f.host = (double *)p;
  if (upload) {
    double2 *aos = f.dev + 4 * 9 * (size_t)g.V;
    for (int d = 0; d < 4; d++) {
      QS_CUDA(cudaMemcpyAsync(aos, p + (size_t)d * 18 * g.V, per, cudaMemcpyHostToDevice, stream()));
      int rc = aos_to_soa((const double *)aos, f.dev + (size_t)d * 9 * g.V, g.V, g.V, 9);
      if (rc) return rc;
    }
  }
  return QEXSTAG_OK;
}

static int field_out(Field4 &f) {
  if (!f.own) return QEXSTAG_OK;
  const Geom &g = *f.g;
  const size_t per = sizeof(double2) * 9 * (size_t)g.V;
  double2 *aos = f.dev + 4 * 9 * (size_t)g.V;
  for (int d = 0; d < 4; d++) {
    int rc = soa_to_aos(f.dev + (size_t)d * 9 * g.V, (double *)aos, g.V, g.V, 9);
    if (rc) return rc;
    QS_CUDA(cudaMemcpyAsync(f.host + (size_t)d * 18 * g.V, aos, per, cudaMemcpyDeviceToHost, stream()));
  }
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

static int check_common(const qexstag_layout *l, int mem) {
  if (!l) return fail(QEXSTAG_ERR_ARG, "null layout");
  if (mem != QEXSTAG_MEM_HOST && mem != QEXSTAG_MEM_DEVICE) return fail(QEXSTAG_ERR_ARG, "bad memory kind");
  return runtime_ready();
}

static int read_results(int n, double *out) {
  QS_CUDA(cudaMemcpyAsync(host_results(), red_results(), sizeof(double) * n, cudaMemcpyDeviceToHost, stream()));
  QS_CUDA(cudaStreamSynchronize(stream()));
  for (int i = 0; i < n; i++) out[i] = host_results()[i];
  return QEXSTAG_OK;
}

}  // namespace qs

using namespace qs;

extern "C" {

void qexstag_gauge_coefs_rect(qexstag_gauge_coefs *c, double beta, double c1) {
  if (!c) return;
  c->plaq = (1.0 - 8.0 * c1) * beta;
  c->rect = c1 * beta;
}

int qexstag_gauge_action(qexstag_layout *l, const qexstag_gauge_coefs *c, const double *u, int mem, double *action) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!c || !u || !action) return fail(QEXSTAG_ERR_ARG, "gauge_action: null argument");
  const Geom &g = l->g;
  Field4 U;
  if ((rc = field_in(g, u, mem, true, U))) return rc;
  const int grid = std::min(grid_for(g.V, kBlock, 8), kMaxRedBlocks * 8 / 2);
  gauge_action_kernel<<<grid, kBlock, 0, stream()>>>(g, U.dev, c->rect != 0.0 ? 1 : 0, red_partials(),
                                                     red_tickets(), red_results());
  note_launch();
  QS_LAUNCH_CHECK();
  double s[2];
  if ((rc = read_results(2, s))) return rc;
  *action = -(c->plaq * s[0] + c->rect * s[1]) / 3.0;
  return QEXSTAG_OK;
}

int qexstag_gauge_force(qexstag_layout *l, const qexstag_gauge_coefs *c, const double *u, double *f, int mem) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!c || !u || !f) return fail(QEXSTAG_ERR_ARG, "gauge_force: null argument");
  const Geom &g = l->g;
  Field4 U, Fo;
  if ((rc = field_in(g, u, mem, true, U)) || (rc = field_in(g, f, mem, false, Fo))) return rc;
  rc = c->rect != 0.0 ? rect_force_dev(l, U.dev, Fo.dev, c->plaq / 3.0, c->rect / 3.0) : QEXSTAG_ERR_ALLOC;
  if (rc == QEXSTAG_ERR_ALLOC) {
    gauge_force_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(g, U.dev, Fo.dev, c->plaq / 3.0, c->rect / 3.0);
    note_launch();
    QS_LAUNCH_CHECK();
  } else if (rc) {
    return rc;
  }
  if ((rc = field_out(Fo))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_link_update(qexstag_layout *l, double *u, const double *p, double eps, int mem) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!u || !p) return fail(QEXSTAG_ERR_ARG, "link_update: null argument");
  if (!std::isfinite(eps)) return fail(QEXSTAG_ERR_ARG, "link_update: eps not finite");
  const Geom &g = l->g;
  Field4 U, P;
  if ((rc = field_in(g, u, mem, true, U)) || (rc = field_in(g, p, mem, true, P))) return rc;
  link_update_kernel<<<field_grid(g), kSmBlock, 0, stream()>>>(g.V, U.dev, P.dev, eps);
  note_launch();
  QS_LAUNCH_CHECK();
  if ((rc = field_out(U))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_momenta_update(qexstag_layout *l, double *p, const double *f, double a, int mem) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!p || !f) return fail(QEXSTAG_ERR_ARG, "momenta_update: null argument");
  const Geom &g = l->g;
  Field4 P, Fi;
  if ((rc = field_in(g, p, mem, true, P)) || (rc = field_in(g, f, mem, true, Fi))) return rc;
  const size_t n = (size_t)36 * g.V;
  axpy_field_kernel<<<grid_for((long)std::min<size_t>(n, 1u << 30)), kBlock, 0, stream()>>>(n, P.dev, a, Fi.dev);
  note_launch();
  QS_LAUNCH_CHECK();
  if ((rc = field_out(P))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_momenta_heatbath(qexstag_layout *l, double *p, unsigned long long seed, unsigned long long counter,
                             int mem) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!p) return fail(QEXSTAG_ERR_ARG, "momenta_heatbath: null argument");
  const Geom &g = l->g;
  if ((long long)4 * g.V > 0xffffffffll) return fail(QEXSTAG_ERR_ARG, "momenta_heatbath: lattice too large");
  Field4 P;
  if ((rc = field_in(g, p, mem, false, P))) return rc;
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  momenta_heatbath_kernel<<<field_grid(g), kSmBlock, 0, stream()>>>(g.V, P.dev, key, (uint32_t)counter,
                                                                    (uint32_t)(counter >> 32));
  note_launch();
  QS_LAUNCH_CHECK();
  if ((rc = field_out(P))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_kinetic_action(qexstag_layout *l, const double *p, int mem, double *t) {
  int rc;
  if ((rc = check_common(l, mem))) return rc;
  if (!p || !t) return fail(QEXSTAG_ERR_ARG, "kinetic_action: null argument");
  const Geom &g = l->g;
  Field4 P;
  if ((rc = field_in(g, p, mem, true, P))) return rc;
  const size_t n = (size_t)36 * g.V;
  const int grid = std::min(grid_for((long)std::min<size_t>(n, 1u << 30), kBlock, 8), kMaxRedBlocks * 8);
  norm2_field_kernel<<<grid, kBlock, 0, stream()>>>(n, P.dev, red_partials(), red_tickets(), red_results());
  note_launch();
  QS_LAUNCH_CHECK();
  double s;
  if ((rc = read_results(1, &s))) return rc;
  *t = 0.5 * s - 16.0 * (double)g.V;
  return QEXSTAG_OK;
}

}  // extern "C"
