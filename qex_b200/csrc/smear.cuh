// smear.cuh -- device helpers and host plumbing shared by the HISQ smearing
// kernels (smear.cu) and their chain rule (smear_deriv.cu).  Fields are
// double2[4][9][V] (direction, element 3*row+col, site index of the QEX V=1
// layout), the library's FP64 link layout.
#pragma once
#include <cmath>
#include <cstring>
#include <new>

#include "lib.cuh"

namespace qs {

int build_low_links(qexstag_links_s *g);

constexpr int kSmBlock = 128;

struct M3 {
  double2 e[9];
};

__device__ __forceinline__ void m_load(M3 &m, const double2 *f, size_t V, int s) {
#pragma unroll
  for (int e = 0; e < 9; e++) m.e[e] = __ldg(f + (size_t)e * V + s);
}
// a matrix of a field that this launch writes: not through the read-only path,
// which is for data that stay as they are while a kernel runs
__device__ __forceinline__ void m_load_own(M3 &m, const double2 *f, size_t V, int s) {
#pragma unroll
  for (int e = 0; e < 9; e++) m.e[e] = f[(size_t)e * V + s];
}
__device__ __forceinline__ void m_store(double2 *f, size_t V, int s, const M3 &m) {
#pragma unroll
  for (int e = 0; e < 9; e++) f[(size_t)e * V + s] = m.e[e];
}
__device__ __forceinline__ void m_axpy(M3 &y, double a, const M3 &x) {
#pragma unroll
  for (int e = 0; e < 9; e++) {
    y.e[e].x = fma(a, x.e[e].x, y.e[e].x);
    y.e[e].y = fma(a, x.e[e].y, y.e[e].y);
  }
}
__device__ __forceinline__ void m_scale(M3 &y, double a) {
#pragma unroll
  for (int e = 0; e < 9; e++) {
    y.e[e].x *= a;
    y.e[e].y *= a;
  }
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// r = a b (registers)
__device__ __forceinline__ void m_nn(M3 &r, const M3 &a, const M3 &b) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 3; k++) s = cmadd(s, a.e[3 * i + k], b.e[3 * k + j]);
      r.e[3 * i + j] = s;
    }
}
// r = a^dag b (registers)
__device__ __forceinline__ void m_dn(M3 &r, const M3 &a, const M3 &b) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 3; k++) s = cjmadd(s, a.e[3 * k + i], b.e[3 * k + j]);
      r.e[3 * i + j] = s;
    }
}

// Site index of x + a*mu (periodic): lex moves by the wrapped step, the
// parity flips with a odd (all L even).
__device__ __forceinline__ int disp1(const Geom &g, const int x[4], int lex, int par, int mu, int a) {
  const int l = lex + lex_step(g, x, mu, a);
  return (l >> 1) + (((par ^ a) & 1) ? g.nh : 0);
}
// x + a*mu + b*nu, mu != nu
__device__ __forceinline__ int disp2(const Geom &g, const int x[4], int lex, int par, int mu, int a, int nu,
                                     int b) {
  const int l = lex + lex_step(g, x, mu, a) + lex_step(g, x, nu, b);
  return (l >> 1) + (((par ^ a ^ b) & 1) ? g.nh : 0);
}

struct SiteCtx {
  int x[4], lex, par, site, mu;
};

// Block b works on direction b % 4 and both parities of the kSmBlock / 2
// half-lattice sites of chunk b / 4, a warp on 32 of one parity.  The four
// blocks that read each other's links as neighbours run together, so those
// reads hit L2 (with the direction-major order every link is fetched from HBM
// again by a later pass), and the sites next to a warp's in x belong to the
// warp beside it, so some of them hit L1: these sweeps are bound by what L2
// delivers to the SMs (12.6 TB/s measured).  Against one parity per block at
// 32^4: staples 814 -> 789 us, middle fields 1972 -> 1905 us.
__device__ __forceinline__ bool site_of_thread(const Geom &g, SiteCtx &c) {
  const int b = blockIdx.x;
  c.mu = b & 3;
  const int w = threadIdx.x >> 5;
  c.par = w & 1;
  const int k = (b >> 2) * (kSmBlock / 2) + (w >> 1) * 32 + (threadIdx.x & 31);
  if (k >= g.nh) return false;
  c.site = c.par * g.nh + k;
  site_coords(g, c.par, k, c.x, c.lex);
  return true;
}

__device__ __forceinline__ void m_zero(M3 &m) {
#pragma unroll
  for (int e = 0; e < 9; e++) m.e[e] = make_double2(0.0, 0.0);
}
// r = a b^dag (registers)
__device__ __forceinline__ void m_nd(M3 &r, const M3 &a, const M3 &b) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 3; k++) s = cjmadd(s, b.e[3 * j + k], a.e[3 * i + k]);
      r.e[3 * i + j] = s;
    }
}

// acc += coef (A B) C^dag of fields A, B, C at sites sa, sb, sc; operands
// streamed a column / row at a time, so that only the partial product and
// acc are live 3x3 matrices
__device__ __forceinline__ void acc_nn_nd(M3 &acc, double coef, const double2 *__restrict__ A, int sa,
                                          const double2 *__restrict__ B, int sb, const double2 *__restrict__ C,
                                          int sc, size_t V) {
  M3 t;
  m_zero(t);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 a[3], b[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      a[j] = __ldg(A + (size_t)(3 * j + k) * V + sa);
      b[j] = __ldg(B + (size_t)(3 * k + j) * V + sb);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) t.e[3 * i + j] = cmadd(t.e[3 * i + j], a[i], b[j]);
  }
#pragma unroll
  for (int j = 0; j < 3; j++) {
    double2 c[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      c[k] = __ldg(C + (size_t)(3 * j + k) * V + sc);
      c[k].x *= coef;
      c[k].y *= coef;
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int k = 0; k < 3; k++) acc.e[3 * i + j] = cjmadd(acc.e[3 * i + j], c[k], t.e[3 * i + k]);
  }
}

// acc += coef (A^dag B) C
__device__ __forceinline__ void acc_dn_nn(M3 &acc, double coef, const double2 *__restrict__ A, int sa,
                                          const double2 *__restrict__ B, int sb, const double2 *__restrict__ C,
                                          int sc, size_t V) {
  M3 t;
  m_zero(t);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 a[3], b[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      a[j] = __ldg(A + (size_t)(3 * k + j) * V + sa);
      b[j] = __ldg(B + (size_t)(3 * k + j) * V + sb);
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) t.e[3 * i + j] = cjmadd(t.e[3 * i + j], a[i], b[j]);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 c[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      c[j] = __ldg(C + (size_t)(3 * k + j) * V + sc);
      c[j].x *= coef;
      c[j].y *= coef;
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) acc.e[3 * i + j] = cmadd(acc.e[3 * i + j], t.e[3 * i + k], c[j]);
  }
}

// acc += coef St_nu(F), the staple of F along nu for link direction mu:
// U_nu(x) F(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag F(x-nu) U_nu(x-nu+mu)
__device__ __forceinline__ void staple_acc(M3 &acc, double coef, const Geom &g, const SiteCtx &c, int mu, int nu,
                                           const double2 *__restrict__ Un, const double2 *__restrict__ F) {
  const size_t V = (size_t)g.V;
  const int s_pn = disp1(g, c.x, c.lex, c.par, nu, 1);
  const int s_pm = disp1(g, c.x, c.lex, c.par, mu, 1);
  const int s_mn = disp1(g, c.x, c.lex, c.par, nu, -1);
  const int s_mnpm = disp2(g, c.x, c.lex, c.par, nu, -1, mu, 1);
  acc_nn_nd(acc, coef, Un, c.site, F, s_pn, Un, s_pm, V);
  acc_dn_nn(acc, coef, Un, s_mn, F, s_mn, Un, s_mnpm, V);
}

__device__ __forceinline__ int other_dir(int mu, int j) { return j < mu ? j : j + 1; }
// index j of direction d among the three directions other than mu
__device__ __forceinline__ int other_index(int mu, int d) { return d < mu ? d : d - 1; }
// field k of an array of link fields
__device__ __forceinline__ size_t fld(const Geom &g, int k) { return (size_t)k * 9 * g.V; }
// r-th direction (r = 0, 1) not in {mu, nu}
__device__ __forceinline__ int third_dir(int mu, int nu, int r) {
  int d = 0, n = 0;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k != mu && k != nu) {
      if (n == r) d = k;
      n++;
    }
  return d;
}

// Re det of a Hermitian matrix (cofactors along row 0)
__device__ __forceinline__ double re_det(const M3 &t) {
  const double2 *m = t.e;
  const double2 c0 = make_double2(cmul(m[4], m[8]).x - cmul(m[5], m[7]).x, cmul(m[4], m[8]).y - cmul(m[5], m[7]).y);
  const double2 c1 = make_double2(cmul(m[5], m[6]).x - cmul(m[3], m[8]).x, cmul(m[5], m[6]).y - cmul(m[3], m[8]).y);
  const double2 c2 = make_double2(cmul(m[3], m[7]).x - cmul(m[4], m[6]).x, cmul(m[3], m[7]).y - cmul(m[4], m[6]).y);
  return cmul(m[0], c0).x + cmul(m[1], c1).x + cmul(m[2], c2).x;
}

// Z = (X^dag X + eps)^(-1/2) and W = X Z.  The inverse square root of the Hermitian
// H = X^dag X + eps is the quadratic c0 + c1 H + c2 H^2 that takes the value
// 1/sqrt(l) at each eigenvalue l (Cayley-Hamilton); the eigenvalues come from
// the trigonometric solution of the characteristic cubic in tr H, tr H^2 and
// det H, as QEX's projectU does.
__device__ __forceinline__ void rsqrt_xdx(M3 &z, const M3 &x, double eps) {
  M3 h, h2;
  m_dn(h, x, x);
  h.e[0].x += eps;
  h.e[4].x += eps;
  h.e[8].x += eps;
  m_nn(h2, h, h);
  const double tr = h.e[0].x + h.e[4].x + h.e[8].x;
  const double p2 = h2.e[0].x + h2.e[4].x + h2.e[8].x;
  const double det = re_det(h);
  const double tr3 = tr * (1.0 / 3.0), tr32 = tr3 * tr3;
  const double q = fabs(0.5 * (p2 * (1.0 / 3.0) - tr32));
  const double r = 0.25 * tr3 * (5.0 * tr32 - p2) - 0.5 * det;
  const double sq = sqrt(q);
  const double isq3 = fmin(3e38, 1.0 / (q * sq));
  const double rs = fmax(-1.0, fmin(1.0, r * isq3));
  const double th = acos(rs) * (1.0 / 3.0);
  double st, ct;
  sincos(th, &st, &ct);
  const double sqc = sq * ct, sqs = 1.7320508075688772 * sq * st;
  const double l0 = tr3 - 2.0 * sqc, l1 = tr3 + sqc + sqs, l2 = tr3 + sqc - sqs;
  const double s0 = sqrt(fabs(l0)), s1 = sqrt(fabs(l1)), s2 = sqrt(fabs(l2));
  const double us = s0 + s1 + s2, ws = s0 * s1 * s2;
  const double di = 1.0 / (ws * (s0 + s1) * (s0 + s2) * (s1 + s2));
  const double c0 = (ws * us * us + l0 * s0 * (l1 + l2) + l1 * s1 * (l0 + l2) + l2 * s2 * (l0 + l1)) * di;
  const double c1 = -(tr * us + ws) * di, c2 = us * di;
#pragma unroll
  for (int e = 0; e < 9; e++) z.e[e] = make_double2(c1 * h.e[e].x + c2 * h2.e[e].x, c1 * h.e[e].y + c2 * h2.e[e].y);
  z.e[0].x += c0;
  z.e[4].x += c0;
  z.e[8].x += c0;
}
__device__ __forceinline__ void project_u(M3 &w, const M3 &x, double eps) {
  M3 z;
  rsqrt_xdx(z, x, eps);
  m_nn(w, x, z);
}

inline dim3 sweep_grid(const Geom &g) { return dim3((unsigned)(4 * ((g.nh + kSmBlock / 2 - 1) / (kSmBlock / 2))), 1, 1); }
inline dim3 field_grid(const Geom &g) { return dim3((unsigned)((g.V + kSmBlock - 1) / kSmBlock), 4, 1); }

// makeImpLinks on device fields: u (stride ufs between directions) -> fl
// (stride ffs); s3 and gm ([4][3][9][V] each) receive the 3-staples and the
// middle fields of the outer staples (null when the level has none)
int fat7_dev(const Geom &g, const qexstag_fat7_coefs &c, const double2 *u, size_t ufs, double2 *fl, size_t ffs,
             double2 *s3, double2 *gm);
// the level's 3-staples and middle fields alone (a level with five-link terms)
int fat7_inner_dev(const Geom &g, const qexstag_fat7_coefs &c, const double2 *u, size_t ufs, double2 *s3,
                   double2 *gm);
// out[mu][j] = St_nu(f_mu), nu = other_dir(mu, j), staples with the links u
int staples_dev(const Geom &g, const double2 *u, size_t ufs, const double2 *f, size_t fs, double2 *out);
// out[mu][j] = c0 base_mu + cl f[mu][j] + c5 (f[mu][a] + f[mu][b])
//              + c7 (St_b(f[mu][a]) + St_a(f[mu][b])), a and b the other two
int mid_dev(const Geom &g, const double2 *u, size_t ufs, double c0, const double2 *base, size_t bs, double cl,
            double c5, double c7, const double2 *f, double2 *out);
int naik_dev(const Geom &g, const double2 *u, size_t ufs, double2 *ll, size_t lfs, double naik);
int project_u_dev(const Geom &g, const double2 *in, size_t ifs, double2 *out, size_t ofs, double eps);

}  // namespace qs

// A smearing handle: the layout and the device scratch of the sweeps.
struct qexstag_smear_s {
  qexstag_layout_s *l = nullptr;
  qs::Workspace ws;
};

namespace qs {

enum SmearSlot { kSmS3 = 0, kSmG, kSmT1, kSmW, kSmIn0, kSmIn1, kSmOut0, kSmOut1, kSmAos };

inline size_t field4_bytes(const Geom &g) { return sizeof(double2) * 9 * (size_t)g.V * 4; }

// device view of a 4-direction gauge field given in either memory space
inline int smear_in(qexstag_smear_s *s, int slot, const double *p, int mem, const double2 **dev) {
  const Geom &g = s->l->g;
  if (mem == QEXSTAG_MEM_DEVICE) {
    *dev = (const double2 *)p;
    return QEXSTAG_OK;
  }
  void *soa, *aos;
  const size_t per = sizeof(double2) * 9 * (size_t)g.V;
  int rc;
  if ((rc = s->ws.get(slot, 4 * per, &soa)) || (rc = s->ws.get(kSmAos, per, &aos))) return rc;
  for (int d = 0; d < 4; d++) {
    QS_CUDA(cudaMemcpyAsync(aos, p + (size_t)d * 18 * g.V, per, cudaMemcpyHostToDevice, stream()));
    if ((rc = aos_to_soa((const double *)aos, (double2 *)soa + (size_t)d * 9 * g.V, g.V, g.V, 9))) return rc;
  }
  *dev = (const double2 *)soa;
  return QEXSTAG_OK;
}

inline int smear_out_buf(qexstag_smear_s *s, int slot, double *p, int mem, double2 **dev) {
  if (mem == QEXSTAG_MEM_DEVICE) {
    *dev = (double2 *)p;
    return QEXSTAG_OK;
  }
  void *soa;
  int rc = s->ws.get(slot, field4_bytes(s->l->g), &soa);
  if (rc) return rc;
  *dev = (double2 *)soa;
  return QEXSTAG_OK;
}

inline int smear_out_finish(qexstag_smear_s *s, const double2 *dev, double *p, int mem) {
  if (mem == QEXSTAG_MEM_DEVICE) return QEXSTAG_OK;
  const Geom &g = s->l->g;
  const size_t per = sizeof(double2) * 9 * (size_t)g.V;
  void *aos;
  int rc = s->ws.get(kSmAos, per, &aos);
  if (rc) return rc;
  for (int d = 0; d < 4; d++) {
    if ((rc = soa_to_aos(dev + (size_t)d * 9 * g.V, (double *)aos, g.V, g.V, 9))) return rc;
    QS_CUDA(cudaMemcpyAsync(p + (size_t)d * 18 * g.V, aos, per, cudaMemcpyDeviceToHost, stream()));
  }
  return QEXSTAG_OK;
}

// a level with Lepage, 5- or 7-staple terms: the outer staples are of other
// fields than U itself
inline bool has_inner(const qexstag_fat7_coefs &c) {
  return c.five_staple != 0.0 || c.seven_staple != 0.0 || c.lepage != 0.0;
}
// a level whose links are side links of staples
inline bool has_side(const qexstag_fat7_coefs &c) { return has_inner(c) || c.three_staple != 0.0; }
inline int smear_scratch(qexstag_smear_s *s, const qexstag_fat7_coefs &c, double2 **s3, double2 **gm) {
  const Geom &g = s->l->g;
  const size_t f = sizeof(double2) * 9 * (size_t)g.V;
  void *p3 = nullptr, *pg = nullptr;
  int rc;
  if (has_inner(c) && ((rc = s->ws.get(kSmS3, 12 * f, &p3)) || (rc = s->ws.get(kSmG, 12 * f, &pg)))) return rc;
  *s3 = (double2 *)p3;
  *gm = (double2 *)pg;
  return QEXSTAG_OK;
}

inline int check_smear(const qexstag_smear_s *s, int mem) {
  if (!s || !s->l) return fail(QEXSTAG_ERR_ARG, "null or destroyed smearing handle");
  if (mem != QEXSTAG_MEM_HOST && mem != QEXSTAG_MEM_DEVICE) return fail(QEXSTAG_ERR_ARG, "bad memory kind");
  return runtime_ready();
}

inline bool finite_coefs(const qexstag_fat7_coefs &c) {
  return std::isfinite(c.one_link) && std::isfinite(c.three_staple) && std::isfinite(c.five_staple) &&
         std::isfinite(c.seven_staple) && std::isfinite(c.lepage);
}

// HisqCoefs.smear of device links g into fat (stride ffs) and long (stride lfs)
int hisq_dev(qexstag_smear_s *s, const qexstag_hisq_coefs &c, const double2 *g, double2 *fat, size_t ffs,
             double2 *lng, size_t lfs);

}  // namespace qs
