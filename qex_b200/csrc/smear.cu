// smear.cu -- HISQ link smearing on the device: QEX's makeImpLinks (fat7 with
// Lepage and Naik terms, src/gauge/fat7l.nim:24-154), projectU
// (src/maths/matrixFunctions.nim:118-212, 340-351) and HisqCoefs.smear
// (src/physics/hisqLinks.nim:40-46).
//
// QEX builds the staples field by field: for each (mu, nu) a 3-staple field,
// then Lepage, 5- and 7-staples from shifted copies of it, about 70 field
// sweeps per level and 18 staples per direction.  The staple of a field F
// along nu, for the link direction mu,
//   St_nu(F) = U_nu(x) F(x+nu) U_nu(x+mu)^dag + U_nu(x-nu)^dag F(x-nu) U_nu(x-nu+mu)
// (computeGenStaple) is linear in F, so the terms that end in a staple along
// the same nu share it (Horner's rule):
//   S_nu = St_nu(U_mu)
//   G_nu = c3 U_mu + cL S_nu + c5 (S_a + S_b) + c7 (St_b(S_a) + St_a(S_b))
//   fl   = c1' U_mu + sum_nu St_nu(G_nu),      {a, b} = the other two directions
// which is 12 staples per direction.  One thread per (site, direction mu)
// and three sweeps: the 12 S fields, the 12 G fields (S read, G written
// once), and fl: 9216 B and 48 staples per site where a field per staple
// took 14976 B and 72.  At 32^4 the whole HISQ smear went from 13.03 to
// 8.74 ms in runs of hundreds, which the power cap holds at 1.6 GHz, and from 11.8
// to 7.7 ms in bursts at 1.965 GHz.  The unitary projection and the Naik product
// naik U(x) U(x+mu) U(x+2mu) are one more sweep each.
//
// Fields are double2[4][9][V] (direction, element 3*row+col, site index of
// the QEX V=1 layout), the library's FP64 link layout.
#include "smear.cuh"

namespace qs {

// out[mu][j] = St_nu(f_mu), nu = other_dir(mu, j): one thread per (site, nu),
// which goes through the three mu with the same links along nu (32^4: 751 us,
// against 789 us for a thread per (site, mu) going through the nu)
__global__ void __launch_bounds__(kSmBlock, 3)
    staples_kernel(const Geom g, const double2 *__restrict__ u, size_t ufs, const double2 *__restrict__ f, size_t fs,
                   double2 *__restrict__ out) {
  SiteCtx c;
  if (!site_of_thread(g, c)) return;
  const int nu = c.mu;
  const size_t V = (size_t)g.V;
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    const int mu = other_dir(nu, j);
    M3 S;
    m_zero(S);
    staple_acc(S, 1.0, g, c, mu, nu, u + nu * ufs, f + mu * fs);
    m_store(out + fld(g, mu * 3 + other_index(mu, nu)), V, c.site, S);
  }
}
struct MidArgs {
  Geom g;
  const double2 *u;
  size_t ufs;
  const double2 *base;
  size_t bs;
  const double2 *f;
  double2 *out;
  double c0, cl, c5, c7;
};

// out[mu][j] = c0 base_mu + cl f[mu][j] + c5 (f[mu][a] + f[mu][b])
//              + c7 (St_b(f[mu][a]) + St_a(f[mu][b]))
__global__ void __launch_bounds__(kSmBlock, 3) mid_kernel(const MidArgs A) {
  SiteCtx c;
  if (!site_of_thread(A.g, c)) return;
  const int mu = c.mu;
  const size_t V = (size_t)A.g.V;
#pragma unroll 1
  for (int j = 0; j < 3; j++) {
    const int rho = other_dir(mu, j);
    const int a = third_dir(mu, rho, 0), b = third_dir(mu, rho, 1);
    const double2 *Fj = A.f + fld(A.g, mu * 3 + j);
    const double2 *Fa = A.f + fld(A.g, mu * 3 + other_index(mu, a));
    const double2 *Fb = A.f + fld(A.g, mu * 3 + other_index(mu, b));
    M3 S, t;
    m_zero(S);
    if (A.c0 != 0.0) {
      m_load(t, A.base + mu * A.bs, V, c.site);
      m_axpy(S, A.c0, t);
    }
    if (A.cl != 0.0) {
      m_load(t, Fj, V, c.site);
      m_axpy(S, A.cl, t);
    }
    if (A.c5 != 0.0) {
      m_load(t, Fa, V, c.site);
      m_axpy(S, A.c5, t);
      m_load(t, Fb, V, c.site);
      m_axpy(S, A.c5, t);
    }
    if (A.c7 != 0.0) {
      staple_acc(S, A.c7, A.g, c, mu, b, A.u + b * A.ufs, Fa);
      staple_acc(S, A.c7, A.g, c, mu, a, A.u + a * A.ufs, Fb);
    }
    m_store(A.out + fld(A.g, mu * 3 + j), V, c.site, S);
  }
}

// fl_mu = c1 U_mu + cs sum_j St_nu(F), F = gm[mu][j], or U_mu itself where gm is null
__global__ void __launch_bounds__(kSmBlock, 3)
    outer_kernel(const Geom g, const double2 *__restrict__ u, size_t ufs, double c1, double cs,
                 const double2 *__restrict__ gm, double2 *__restrict__ fl, size_t ffs) {
  SiteCtx c;
  if (!site_of_thread(g, c)) return;
  const int mu = c.mu;
  const size_t V = (size_t)g.V;
  const double2 *Um = u + mu * ufs;
  M3 acc;
  m_load(acc, Um, V, c.site);
  m_scale(acc, c1);
  if (cs != 0.0) {
#pragma unroll 1
    for (int j = 0; j < 3; j++) {
      const int nu = other_dir(mu, j);
      staple_acc(acc, cs, g, c, mu, nu, u + nu * ufs, gm ? gm + fld(g, mu * 3 + j) : Um);
    }
  }
  m_store(fl + mu * ffs, V, c.site, acc);
}

// ll_mu(x) = naik U_mu(x) (U_mu(x+mu) U_mu(x+2mu))   (fat7l.nim:142-154)
__global__ void __launch_bounds__(kSmBlock)
    naik_kernel(Geom g, const double2 *__restrict__ u, size_t ufs, double2 *ll, size_t lfs, double naik) {
  SiteCtx c;
  if (!site_of_thread(g, c)) return;
  const int mu = c.mu;
  const size_t V = (size_t)g.V;
  const double2 *U = u + mu * ufs;
  M3 a, b, t;
  m_load(a, U, V, disp1(g, c.x, c.lex, c.par, mu, 1));
  m_load(b, U, V, disp1(g, c.x, c.lex, c.par, mu, 2));
  m_nn(t, a, b);
  m_load(a, U, V, c.site);
  m_nn(b, a, t);
  m_scale(b, naik);
  m_store(ll + mu * lfs, V, c.site, b);
}

__global__ void __launch_bounds__(kSmBlock)
    project_u_kernel(int V, const double2 *__restrict__ in, size_t ifs, double2 *out, size_t ofs, double eps) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const int mu = blockIdx.y;
  M3 x, w;
  m_load(x, in + mu * ifs, (size_t)V, s);
  project_u(w, x, eps);
  m_store(out + mu * ofs, (size_t)V, s, w);
}

int staples_dev(const Geom &g, const double2 *u, size_t ufs, const double2 *f, size_t fs, double2 *out) {
  staples_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(g, u, ufs, f, fs, out);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

int mid_dev(const Geom &g, const double2 *u, size_t ufs, double c0, const double2 *base, size_t bs, double cl,
            double c5, double c7, const double2 *f, double2 *out) {
  mid_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(MidArgs{g, u, ufs, base, bs, f, out, c0, cl, c5, c7});
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

int fat7_inner_dev(const Geom &g, const qexstag_fat7_coefs &c, const double2 *u, size_t ufs, double2 *s3,
                   double2 *gm) {
  int rc = staples_dev(g, u, ufs, u, ufs, s3);
  if (rc) return rc;
  return mid_dev(g, u, ufs, c.three_staple, u, ufs, c.lepage, c.five_staple, c.seven_staple, s3, gm);
}

int fat7_dev(const Geom &g, const qexstag_fat7_coefs &c, const double2 *u, size_t ufs, double2 *fl, size_t ffs,
             double2 *s3, double2 *gm) {
  const bool inner = has_inner(c);
  int rc;
  if (inner && (rc = fat7_inner_dev(g, c, u, ufs, s3, gm))) return rc;
  outer_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(g, u, ufs, c.one_link - 6.0 * c.lepage,
                                                         inner ? 1.0 : c.three_staple, inner ? gm : nullptr, fl, ffs);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

int naik_dev(const Geom &g, const double2 *u, size_t ufs, double2 *ll, size_t lfs, double naik) {
  naik_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(g, u, ufs, ll, lfs, naik);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

int project_u_dev(const Geom &g, const double2 *in, size_t ifs, double2 *out, size_t ofs, double eps) {
  project_u_kernel<<<field_grid(g), kSmBlock, 0, stream()>>>(g.V, in, ifs, out, ofs, eps);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

}  // namespace qs

namespace qs {

// HisqCoefs.smear into device fields fat (stride ffs) and long (stride lfs)
int hisq_dev(qexstag_smear_s *s, const qexstag_hisq_coefs &c, const double2 *g, double2 *fat, size_t ffs,
             double2 *lng, size_t lfs) {
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  void *pt1, *pw;
  double2 *s3, *gm;
  int rc;
  if ((rc = s->ws.get(kSmT1, field4_bytes(geo), &pt1)) || (rc = s->ws.get(kSmW, field4_bytes(geo), &pw))) return rc;
  if ((rc = smear_scratch(s, c.fat7first, &s3, &gm)) ||
      (rc = fat7_dev(geo, c.fat7first, g, fs, (double2 *)pt1, fs, s3, gm)))
    return rc;
  if ((rc = project_u_dev(geo, (const double2 *)pt1, fs, (double2 *)pw, fs, c.reunit_eps))) return rc;
  if ((rc = smear_scratch(s, c.fat7second, &s3, &gm)) ||
      (rc = fat7_dev(geo, c.fat7second, (const double2 *)pw, fs, fat, ffs, s3, gm)))
    return rc;
  if (c.naik != 0.0) return naik_dev(geo, (const double2 *)pw, fs, lng, lfs, c.naik);
  // no Naik term: long links are zero
  for (int d = 0; d < 4; d++) QS_CUDA(cudaMemsetAsync(lng + d * lfs, 0, sizeof(double2) * fs, stream()));
  return QEXSTAG_OK;
}

}  // namespace qs

using namespace qs;

extern "C" {

void qexstag_fat7_coefs_set_hisq(qexstag_fat7_coefs *c, double f7lf, double naik) {
  if (!c) return;
  c->one_link = (1.0 + 3.0 * f7lf + naik) / 8.0;
  c->three_staple = -1.0 / 16.0;
  c->five_staple = 1.0 / 64.0;
  c->seven_staple = -1.0 / 384.0;
  c->lepage = -f7lf / 16.0;
}

void qexstag_hisq_coefs_init(qexstag_hisq_coefs *c, double lepage, double naik) {
  if (!c) return;
  std::memset(c, 0, sizeof(*c));
  qexstag_fat7_coefs_set_hisq(&c->fat7first, lepage, 0.0);
  qexstag_fat7_coefs_set_hisq(&c->fat7second, 2.0 - lepage, naik);
  c->naik = -naik / 24.0;
  c->reunit_eps = 1e-20;
}

int qexstag_smear_create(qexstag_layout *l, qexstag_smear **out) {
  if (!l || !out) return fail(QEXSTAG_ERR_ARG, "smear_create: null argument");
  int rc = runtime_ready();
  if (rc) return rc;
  qexstag_smear_s *s = new (std::nothrow) qexstag_smear_s;
  if (!s) return fail(QEXSTAG_ERR_ALLOC, "smear_create: out of host memory");
  s->l = l;
  *out = s;
  return QEXSTAG_OK;
}

int qexstag_smear_destroy(qexstag_smear *s) {
  if (!s) return QEXSTAG_OK;
  s->ws.release();
  s->l = nullptr;
  delete s;
  return QEXSTAG_OK;
}

int qexstag_fat7(qexstag_smear *s, const qexstag_fat7_coefs *c, const double *gf, double *fl,
                 const double *gf_long, double *ll, double naik, int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!c || !gf || !fl) return fail(QEXSTAG_ERR_ARG, "fat7: null argument");
  if (!finite_coefs(*c) || !std::isfinite(naik)) return fail(QEXSTAG_ERR_ARG, "fat7: coefficients not finite");
  const bool want_long = naik != 0.0 && gf_long && ll;
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  const double2 *u, *ul = nullptr;
  double2 *f, *l = nullptr, *s3, *gm;
  if ((rc = smear_in(s, kSmIn0, gf, mem, &u)) || (rc = smear_out_buf(s, kSmOut0, fl, mem, &f))) return rc;
  if (want_long) {
    if (gf_long == gf)
      ul = u;
    else if ((rc = smear_in(s, kSmIn1, gf_long, mem, &ul)))
      return rc;
    if ((rc = smear_out_buf(s, kSmOut1, ll, mem, &l))) return rc;
  }
  if ((rc = smear_scratch(s, *c, &s3, &gm)) || (rc = fat7_dev(geo, *c, u, fs, f, fs, s3, gm))) return rc;
  if (want_long && (rc = naik_dev(geo, ul, fs, l, fs, naik))) return rc;
  if ((rc = smear_out_finish(s, f, fl, mem))) return rc;
  if (want_long && (rc = smear_out_finish(s, l, ll, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_project_u(qexstag_smear *s, const double *x, double *u, double eps, int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!x || !u) return fail(QEXSTAG_ERR_ARG, "project_u: null argument");
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  const double2 *xin;
  double2 *w;
  if ((rc = smear_in(s, kSmIn0, x, mem, &xin)) || (rc = smear_out_buf(s, kSmOut0, u, mem, &w))) return rc;
  if ((rc = project_u_dev(geo, xin, fs, w, fs, eps)) || (rc = smear_out_finish(s, w, u, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_hisq_smear(qexstag_smear *s, const qexstag_hisq_coefs *c, const double *g, double *fat, double *lng,
                       int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!c || !g || !fat || !lng) return fail(QEXSTAG_ERR_ARG, "hisq_smear: null argument");
  if (!finite_coefs(c->fat7first) || !finite_coefs(c->fat7second) || !std::isfinite(c->naik))
    return fail(QEXSTAG_ERR_ARG, "hisq_smear: coefficients not finite");
  const size_t fs = (size_t)9 * s->l->g.V;
  const double2 *u;
  double2 *f, *l;
  if ((rc = smear_in(s, kSmIn0, g, mem, &u)) || (rc = smear_out_buf(s, kSmOut0, fat, mem, &f)) ||
      (rc = smear_out_buf(s, kSmOut1, lng, mem, &l)))
    return rc;
  if ((rc = hisq_dev(s, *c, u, f, fs, l, fs))) return rc;
  if ((rc = smear_out_finish(s, f, fat, mem)) || (rc = smear_out_finish(s, l, lng, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_links_hisq(qexstag_links *g, qexstag_smear *s, const qexstag_hisq_coefs *c, const double *thin,
                       int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!g || !g->u64 || !c || !thin) return fail(QEXSTAG_ERR_ARG, "links_hisq: null argument");
  if (g->nl != 8) return fail(QEXSTAG_ERR_ARG, "links_hisq: the link handle must hold 8 (fat+Naik) links");
  if (g->l != s->l) return fail(QEXSTAG_ERR_ARG, "links_hisq: handles on different layouts");
  if (!finite_coefs(c->fat7first) || !finite_coefs(c->fat7second) || !std::isfinite(c->naik))
    return fail(QEXSTAG_ERR_ARG, "links_hisq: coefficients not finite");
  const size_t fs = (size_t)9 * s->l->g.V;
  const double2 *u;
  if ((rc = smear_in(s, kSmIn0, thin, mem, &u))) return rc;
  // fat link of direction mu at list entry 2 mu, long link at 2 mu + 1
  if ((rc = hisq_dev(s, *c, u, g->u64, 2 * fs, g->u64 + fs, 2 * fs))) return rc;
  if ((rc = build_low_links(g))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

}  // extern "C"
