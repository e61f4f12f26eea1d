// smear_deriv.cu -- the chain rule through HISQ smearing on the device: the
// derivative of S = sum_x Re Tr C(x)^dag out(x) with respect to the input
// links, in QEX's convention dS = sum Re Tr dU^dag f
// (src/gauge/hisqsmear.nim:66-168: smearGetForce and its check).  QEX
// computes it as fat7lDeriv (src/gauge/fat7lderiv.nim:122-331), projectUderiv
// (src/maths/matrixFunctions.nim:368-390) and fat7lDeriv again.
//
// Here each fat7 level, in the form of smear.cu (S_nu = St_nu(U_mu), G_nu,
// fl = c1' U + sum_nu St_nu(G_nu)), is differentiated in four sweeps over
// (site, direction), with S and G from the forward sweeps.  With M the
// chain on the fat links:
//   T_nu  = St_nu(M_mu)                                (chain on G_nu)
//   M3_nu = cL T_nu + c5 (T_a + T_b) + c7 (St_b(T_a) + St_a(T_b))
//                                                      (chain on S_nu)
// are the forward's own first two sweeps run on M, and the last two form
//   dU_d(y) = c1' M_d + sum_nu (c3 T_nu + St_nu(M3_nu))   (U_d the middle link)
//             + the derivatives of the staples in which U_d is a side link,
//               for each other direction mu: the outer staple along d (chain
//               M, middle G_d), the two inner ones (chain c7 T_a, middle
//               S_b, and a, b exchanged) and the 3-staple (chain M3_d,
//               middle U_mu)
//             + the Naik product's three positions.
// St(g; F) = g(x) F(x+nu) g(x+mu)^dag + g(x-nu)^dag F(x-nu) g(x-nu+mu) is the
// staple of the field F along nu; it is also its own adjoint in F, which is
// why the chains on the inner staples are staples of the outer chains.  The
// derivative of St(g1; g2) (side direction d1, link direction d2) with chain c
// with respect to the side field at y is
//   c(y) g1(y+d2) g2(y+d1)^dag + g2(y) g1(y+d2) c(y+d1)^dag
//   + c(y-d2)^dag g1(y-d2) g2(y-d2+d1) + g2(y-d2)^dag g1(y-d2) c(y-d2+d1),
// that is, with z = y-d2, two terms of y's own operands at y and y+d1 and two
// of z's at z and z+d1.  Gathered at y they read every field at four sites.
// Here a thread forms, from its operands at y and y+d1, the two terms of y
// and the two that belong to y+d2; the latter go to a field of their own
// (one per pair of directions) that the last sweep reads: no atomics, and
// half the matrices through L2, which bounds these sweeps.  Chain rule on
// 12 x 20 x 14 x 18: 3.33 ms with up to five fields summed at each gather,
// 2.07 with single fields, 1.87 with the terms formed at their operands.
#include "smear.cuh"

namespace qs {

struct AdjArgs {
  Geom g;
  const double2 *u;   // level input links, direction d at u + d*ufs
  size_t ufs;
  const double2 *m;   // chain on the fat links, stride mfs
  size_t mfs;
  const double2 *lm;  // chain on the long links (nullptr: no Naik term), stride lmfs
  size_t lmfs;
  double naik;
  const double2 *s3;  // [4][3][9][V] forward 3-staples (when the level has inner terms)
  const double2 *gm;  // [4][3][9][V] forward middle fields of the outer staples
  const double2 *t7;  // [4][3][9][V] T
  const double2 *m3;  // [4][3][9][V] M3
  double2 *d;         // output derivative, stride dfs
  size_t dfs;
  int accumulate;     // add to d instead of overwriting it
  double c1, c3, c7;
  int inner, side;
  double2 *q;         // [4][3][9][V] side terms on their way to y + mu
};

// One product of the side derivatives with chain or middle fields A at y and
// B at y + d, g1 the side field's links:
//   p += coef A(y) g1(y+mu) B(y+d)^dag        (belongs to y)
//   q += coef A(y)^dag g1(y) B(y+d)           (belongs to y + mu)
__device__ __forceinline__ void side_term(M3 &p, M3 &q, double coef, const double2 *__restrict__ A, int sy,
                                          const double2 *__restrict__ B, int syd, const double2 *__restrict__ g1,
                                          int symu, size_t V) {
  M3 b, t;
  m_load(b, B, V, syd);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double2 r[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      r[k] = __ldg(g1 + (size_t)(3 * i + k) * V + symu);
      r[k].x *= coef;
      r[k].y *= coef;
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double2 s = make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 3; k++) s = cjmadd(s, b.e[3 * j + k], r[k]);
      t.e[3 * i + j] = s;
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 a[3];
#pragma unroll
    for (int i = 0; i < 3; i++) a[i] = __ldg(A + (size_t)(3 * i + k) * V + sy);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) p.e[3 * i + j] = cmadd(p.e[3 * i + j], a[i], t.e[3 * k + j]);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double2 r[3], u[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
      r[l] = __ldg(g1 + (size_t)(3 * k + l) * V + sy);
      r[l].x *= coef;
      r[l].y *= coef;
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
      u[j] = make_double2(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < 3; l++) u[j] = cmadd(u[j], r[l], b.e[3 * l + j]);
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double2 a = __ldg(A + (size_t)(3 * k + i) * V + sy);
#pragma unroll
      for (int j = 0; j < 3; j++) q.e[3 * i + j] = cjmadd(q.e[3 * i + j], a, u[j]);
    }
  }
}

// the side terms with U_d: those of y go to d_d(y), those of y + mu to
// q[d][mu](y), which the last sweep picks up.  255 registers and 8 warps an
// SM: 306 us on 12 x 20 x 14 x 18, against 371 us at 168 registers and 12
// warps, which spill.
__global__ void __launch_bounds__(kSmBlock, 2) fat7_adj_side_kernel(const AdjArgs A) {
  SiteCtx c;
  if (!site_of_thread(A.g, c)) return;
  const int d = c.mu;
  const Geom &g = A.g;
  const size_t V = (size_t)g.V;
  const double2 *Ud = A.u + d * A.ufs;
  M3 p;
  m_zero(p);
  if (A.accumulate) m_load_own(p, A.d + d * A.dfs, V, c.site);
  const int syd = disp1(g, c.x, c.lex, c.par, d, 1);
#pragma unroll 1
  for (int jm = 0; jm < 3; jm++) {
    const int mu = other_dir(d, jm);
    const int symu = disp1(g, c.x, c.lex, c.par, mu, 1);
    const int ja = mu * 3 + other_index(mu, third_dir(mu, d, 0)), jb = mu * 3 + other_index(mu, third_dir(mu, d, 1));
    const int jd = mu * 3 + other_index(mu, d);
    M3 q;
    m_zero(q);
    const int np = !A.inner ? 1 : A.c7 != 0.0 ? 4 : 2;
#pragma unroll 1
    for (int k = 0; k < 2 * np; k++) {
      // pair k / 2 of chain and middle field, as (chain, middle) and (middle, chain)
      const double2 *C = A.m + mu * A.mfs, *G = A.u + mu * A.ufs;
      double coef = A.c3;
      if (A.inner) {
        const int pr = k >> 1;
        coef = pr < 2 ? 1.0 : A.c7;
        if (pr == 0) G = A.gm + fld(g, jd);
        if (pr == 1) C = A.m3 + fld(g, jd);
        if (pr >= 2) {
          C = A.t7 + fld(g, pr == 2 ? ja : jb);
          G = A.s3 + fld(g, pr == 2 ? jb : ja);
        }
      }
      side_term(p, q, coef, (k & 1) ? G : C, c.site, (k & 1) ? C : G, syd, Ud, symu, V);
    }
    m_store(A.q + fld(g, d * 3 + jm), V, c.site, q);
  }
  m_store(A.d + d * A.dfs, V, c.site, p);
}

// the derivative with respect to U_d at y: the side terms, U_d as the middle
// link, and the Naik product
__global__ void __launch_bounds__(kSmBlock, 3) fat7_adj_link_kernel(const AdjArgs A) {
  SiteCtx c;
  if (!site_of_thread(A.g, c)) return;
  const int d = c.mu;
  const Geom &g = A.g;
  const size_t V = (size_t)g.V;
  const double2 *Ud = A.u + d * A.ufs;
  M3 acc;
  m_zero(acc);
  if (A.accumulate || A.side) m_load_own(acc, A.d + d * A.dfs, V, c.site);
  {
    M3 md;
    m_load(md, A.m + d * A.mfs, V, c.site);
    m_axpy(acc, A.c1, md);
  }
  if (A.side) {
#pragma unroll 1
    for (int j = 0; j < 3; j++) {
      const int nu = other_dir(d, j);
      M3 t;
      m_load(t, A.q + fld(g, d * 3 + j), V, disp1(g, c.x, c.lex, c.par, nu, -1));
      m_axpy(acc, 1.0, t);
      if (A.inner && A.c3 != 0.0) {
        m_load(t, A.t7 + fld(g, d * 3 + j), V, c.site);
        m_axpy(acc, A.c3, t);
      }
      staple_acc(acc, A.inner ? 1.0 : A.c3, g, c, d, nu, A.u + nu * A.ufs,
                 A.inner ? A.m3 + fld(g, d * 3 + j) : A.m + d * A.mfs);
    }
  }
  if (A.lm) {
    // ll_d(x) = naik W(x) W(x+d) W(x+2d), W = U_d: the three positions of y
    const double2 *LM = A.lm + d * A.lmfs;
    const int s_p1 = disp1(g, c.x, c.lex, c.par, d, 1), s_p2 = disp1(g, c.x, c.lex, c.par, d, 2);
    const int s_m1 = disp1(g, c.x, c.lex, c.par, d, -1), s_m2 = disp1(g, c.x, c.lex, c.par, d, -2);
    M3 a, b, t;
    // LM(y) (W(y+d) W(y+2d))^dag
    m_load(a, Ud, V, s_p1);
    m_load(b, Ud, V, s_p2);
    m_nn(t, a, b);
    m_load(a, LM, V, c.site);
    m_nd(b, a, t);
    m_axpy(acc, A.naik, b);
    // W(y-d)^dag LM(y-d) W(y+d)^dag
    m_load(a, Ud, V, s_m1);
    m_load(b, LM, V, s_m1);
    m_dn(t, a, b);
    m_load(a, Ud, V, s_p1);
    m_nd(b, t, a);
    m_axpy(acc, A.naik, b);
    // (W(y-2d) W(y-d))^dag LM(y-2d)
    m_load(a, Ud, V, s_m2);
    m_load(b, Ud, V, s_m1);
    m_nn(t, a, b);
    m_load(a, LM, V, s_m2);
    m_dn(b, t, a);
    m_axpy(acc, A.naik, b);
  }
  m_store(A.d + d * A.dfs, V, c.site, acc);
}

// ---------------------------------------------------------------------------
// projectU's chain rule (matrixFunctions.nim:368-390): U = X Z, Z = (X^dag X +
// eps)^(-1/2), Y = Z^-1; with chain C
//   r = C Z - X (T + T^dag),   Y T + T Y = U^dag C Z
// The Sylvester equation is solved in closed form from the adjugate and the
// invariants of Y (projUderiv.nim:96-145, 3x3 branch).
// ---------------------------------------------------------------------------

__device__ __forceinline__ void m_adjugate(M3 &r, const M3 &x) {
  const double2 *m = x.e;
  auto sub = [](double2 a, double2 b, double2 c, double2 d) {
    const double2 p = cmul(a, b), q = cmul(c, d);
    return make_double2(p.x - q.x, p.y - q.y);
  };
  r.e[0] = sub(m[4], m[8], m[5], m[7]);
  r.e[1] = sub(m[7], m[2], m[8], m[1]);
  r.e[2] = sub(m[1], m[5], m[2], m[4]);
  r.e[3] = sub(m[5], m[6], m[3], m[8]);
  r.e[4] = sub(m[8], m[0], m[6], m[2]);
  r.e[5] = sub(m[2], m[3], m[0], m[5]);
  r.e[6] = sub(m[3], m[7], m[4], m[6]);
  r.e[7] = sub(m[6], m[1], m[7], m[0]);
  r.e[8] = sub(m[0], m[4], m[1], m[3]);
}

// x with a x + x a = c, a Hermitian positive definite (invariants real)
__device__ __forceinline__ void sylsolve3(M3 &x, const M3 &a, const M3 &c) {
  M3 ad, p, q;
  m_adjugate(ad, a);
  const double t = a.e[0].x + a.e[4].x + a.e[8].x;
  const double s = ad.e[0].x + ad.e[4].x + ad.e[8].x;
  const double r = cmul(a.e[0], ad.e[0]).x + cmul(a.e[1], ad.e[3]).x + cmul(a.e[2], ad.e[6]).x;
  const double c2 = 1.0 / (2.0 * (s * t - r));
  const double c0 = c2 * (s + t * t), c1 = c2 * (t / r), c4 = c2 * t;
#pragma unroll
  for (int e = 0; e < 9; e++) x.e[e] = make_double2(c0 * c.e[e].x, c0 * c.e[e].y);
  m_nn(p, a, c);       // a c
  m_axpy(x, -c4, p);
  m_nn(q, p, a);       // a c a
  m_axpy(x, c2, q);
  m_nn(p, c, a);       // c a
  m_axpy(x, -c4, p);
  m_nn(p, ad, c);      // ad c
  m_axpy(x, -c2, p);
  m_nn(q, p, ad);      // ad c ad
  m_axpy(x, c1, q);
  m_nn(p, c, ad);      // c ad
  m_axpy(x, -c2, p);
}

__global__ void __launch_bounds__(kSmBlock)
    project_u_deriv_kernel(int V, const double2 *__restrict__ u, const double2 *__restrict__ x,
                           const double2 *chain, double2 *out, size_t fs, double eps) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const size_t off = blockIdx.y * fs;
  M3 X, Z, Y, R, T;
  m_load(X, x + off, (size_t)V, s);
  rsqrt_xdx(Z, X, eps);
  {
    // Y = Z^-1 = adj(Z) / det Z
    M3 ad;
    m_adjugate(ad, Z);
    const double2 det = make_double2(cmul(Z.e[0], ad.e[0]).x + cmul(Z.e[1], ad.e[3]).x + cmul(Z.e[2], ad.e[6]).x,
                                     cmul(Z.e[0], ad.e[0]).y + cmul(Z.e[1], ad.e[3]).y + cmul(Z.e[2], ad.e[6]).y);
    const double nn = det.x * det.x + det.y * det.y;
    const double2 idet = make_double2(det.x / nn, -det.y / nn);
#pragma unroll
    for (int e = 0; e < 9; e++) Y.e[e] = cmul(ad.e[e], idet);
  }
  m_load_own(T, chain + off, (size_t)V, s);  // out may be chain
  m_nn(R, T, Z);  // C Z
  m_load(T, u + off, (size_t)V, s);
  m_dn(Z, T, R);  // U^dag C Z
  sylsolve3(T, Y, Z);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 a = T.e[3 * i + j], b = T.e[3 * j + i];
      Z.e[3 * i + j] = make_double2(a.x + b.x, a.y - b.y);  // T + T^dag
    }
  m_nn(T, X, Z);
  m_axpy(R, -1.0, T);
  m_store(out + off, (size_t)V, s, R);
}

int project_u_deriv_dev(const Geom &g, const double2 *u, const double2 *x, const double2 *chain, double2 *out,
                        double eps) {
  project_u_deriv_kernel<<<field_grid(g), kSmBlock, 0, stream()>>>(g.V, u, x, chain, out, (size_t)9 * g.V, eps);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// fat7lDeriv on device fields: d (+)= derivative w.r.t. u of
// sum Re Tr (m^dag fat7(u) + lm^dag naik u(x)u(x+mu)u(x+2mu)); s3 and gm hold
// the level's forward fields (fat7_inner_dev on u), t7 and m3 are 12-field
// scratch.
int fat7_adj_dev(const Geom &g, const qexstag_fat7_coefs &c, const double2 *u, size_t ufs, const double2 *m,
                 size_t mfs, const double2 *lm, size_t lmfs, double naik, const double2 *s3, const double2 *gm,
                 double2 *t7, double2 *m3, double2 *q, double2 *d, size_t dfs, bool accumulate) {
  AdjArgs A;
  A.g = g;
  A.u = u;
  A.ufs = ufs;
  A.m = m;
  A.mfs = mfs;
  A.lm = (naik != 0.0) ? lm : nullptr;
  A.lmfs = lmfs;
  A.naik = naik;
  A.s3 = s3;
  A.gm = gm;
  A.t7 = t7;
  A.m3 = m3;
  A.d = d;
  A.dfs = dfs;
  A.accumulate = accumulate ? 1 : 0;
  A.c1 = c.one_link - 6.0 * c.lepage;
  A.c3 = c.three_staple;
  A.c7 = c.seven_staple;
  A.inner = has_inner(c) ? 1 : 0;
  A.side = has_side(c) ? 1 : 0;
  A.q = q;
  int rc;
  if (A.inner && ((rc = staples_dev(g, u, ufs, m, mfs, t7)) ||
                  (rc = mid_dev(g, u, ufs, 0.0, nullptr, 0, c.lepage, c.five_staple, c.seven_staple, t7, m3))))
    return rc;
  if (A.side) {
    fat7_adj_side_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(A);
    note_launch();
  }
  fat7_adj_link_kernel<<<sweep_grid(g), kSmBlock, 0, stream()>>>(A);
  note_launch();
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

enum DerivSlot { kSdT7 = 40, kSdM3, kSdQ, kSdTmp, kSdDW, kSdIn2, kSdIn3 };

// scratch of a level's adjoint (null where the level has no use for it)
static int adj_scratch(qexstag_smear_s *s, const qexstag_fat7_coefs &lv, double2 **t7, double2 **m3, double2 **q) {
  const size_t f = sizeof(double2) * 9 * (size_t)s->l->g.V;
  void *a = nullptr, *b = nullptr, *c = nullptr;
  int rc;
  if (has_inner(lv) && ((rc = s->ws.get(kSdT7, 12 * f, &a)) || (rc = s->ws.get(kSdM3, 12 * f, &b)))) return rc;
  if (has_side(lv) && (rc = s->ws.get(kSdQ, 12 * f, &c))) return rc;
  *t7 = (double2 *)a;
  *m3 = (double2 *)b;
  *q = (double2 *)c;
  return QEXSTAG_OK;
}

// smearGetForce's chain rule on device fields.  forward: the last call on
// this handle's scratch was hisq_dev of the same links, whose projected
// links and second-level fields are used as they are.
static int hisq_deriv_dev(qexstag_smear_s *s, const qexstag_hisq_coefs &c, const double2 *g, const double2 *cf,
                          size_t cfs, const double2 *cl, size_t cls, double2 *d, bool forward) {
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  void *pv, *pw, *pd;
  double2 *s3, *gm, *t7, *m3, *q;
  int rc;
  if ((rc = s->ws.get(kSmT1, field4_bytes(geo), &pv)) || (rc = s->ws.get(kSmW, field4_bytes(geo), &pw)) ||
      (rc = s->ws.get(kSdDW, field4_bytes(geo), &pd)))
    return rc;
  double2 *v = (double2 *)pv, *w = (double2 *)pw, *dw = (double2 *)pd;
  if (!forward) {
    // v = fat7(g), w = projectU(v), and the second level's inner fields
    if ((rc = smear_scratch(s, c.fat7first, &s3, &gm)) || (rc = fat7_dev(geo, c.fat7first, g, fs, v, fs, s3, gm)) ||
        (rc = project_u_dev(geo, v, fs, w, fs, c.reunit_eps)) || (rc = smear_scratch(s, c.fat7second, &s3, &gm)))
      return rc;
    if (has_inner(c.fat7second) && (rc = fat7_inner_dev(geo, c.fat7second, w, fs, s3, gm))) return rc;
  } else if ((rc = smear_scratch(s, c.fat7second, &s3, &gm))) {
    return rc;
  }
  // second level (fat7 and Naik both of w) -> dS/dw
  if ((rc = adj_scratch(s, c.fat7second, &t7, &m3, &q)) ||
      (rc = fat7_adj_dev(geo, c.fat7second, w, fs, cf, cfs, cl, cls, c.naik, s3, gm, t7, m3, q, dw, fs, false)))
    return rc;
  // projectU -> dS/dv (in place)
  if ((rc = project_u_deriv_dev(geo, w, v, dw, dw, c.reunit_eps))) return rc;
  // first level: its inner fields again, then dS/dg
  if ((rc = smear_scratch(s, c.fat7first, &s3, &gm)) || (rc = adj_scratch(s, c.fat7first, &t7, &m3, &q))) return rc;
  if (has_inner(c.fat7first) && (rc = fat7_inner_dev(geo, c.fat7first, g, fs, s3, gm))) return rc;
  return fat7_adj_dev(geo, c.fat7first, g, fs, dw, fs, nullptr, 0, 0.0, s3, gm, t7, m3, q, d, fs, false);
}

// F_d(x) = projectTAH(ff_d(x) U_d(x)^dag)   (fermForce's last step,
// hmcAction.nim:780-790; projectTAH: matrixFunctions.nim:414-419)
__global__ void __launch_bounds__(kSmBlock)
    tah_times_adj_kernel(int V, const double2 *__restrict__ ff, const double2 *__restrict__ u, double2 *out,
                         size_t fs) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= V) return;
  const size_t off = blockIdx.y * fs;
  M3 a, b, m;
  m_load(a, ff + off, (size_t)V, s);
  m_load(b, u + off, (size_t)V, s);
  m_nd(m, a, b);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double2 p = m.e[3 * i + j], q = m.e[3 * j + i];
      a.e[3 * i + j] = make_double2(0.5 * (p.x - q.x), 0.5 * (p.y + q.y));
    }
  const double tr = (a.e[0].y + a.e[4].y + a.e[8].y) * (1.0 / 3.0);
  a.e[0].y -= tr;
  a.e[4].y -= tr;
  a.e[8].y -= tr;
  m_store(out + off, (size_t)V, s, a);
}

enum ForceSlot { kSfPhi = 60, kSfPsi, kSfF8, kSfFF };

}  // namespace qs

using namespace qs;

extern "C" {

int qexstag_fat7_deriv(qexstag_smear *s, const qexstag_fat7_coefs *c, const double *gauge, const double *mid,
                       double *deriv, const double *llgauge, const double *llmid, double *llderiv, double naik,
                       int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!c || !gauge || !mid || !deriv) return fail(QEXSTAG_ERR_ARG, "fat7_deriv: null argument");
  if (!finite_coefs(*c) || !std::isfinite(naik)) return fail(QEXSTAG_ERR_ARG, "fat7_deriv: coefficients not finite");
  const bool want_long = naik != 0.0 && llgauge && llmid && llderiv;
  const bool same = want_long && llgauge == gauge && llderiv == deriv;
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  const double2 *u, *m, *ul = nullptr, *lmid = nullptr, *d0;
  double2 *d, *dl = nullptr, *s3, *gm, *t7, *m3, *q;
  if ((rc = smear_in(s, kSmIn0, gauge, mem, &u)) || (rc = smear_in(s, kSmIn1, mid, mem, &m)) ||
      (rc = smear_in(s, kSdIn2, deriv, mem, &d0)))
    return rc;
  d = (double2 *)d0;  // host: the staged copy is updated and copied back
  if (want_long) {
    if ((rc = smear_in(s, kSdIn3, llmid, mem, &lmid))) return rc;
    if (same) {
      ul = u;
      dl = d;
    } else {
      const double2 *dl0;
      if ((rc = smear_in(s, kSmOut0, llgauge, mem, &ul)) || (rc = smear_in(s, kSmOut1, llderiv, mem, &dl0))) return rc;
      dl = (double2 *)dl0;
    }
  }
  if ((rc = smear_scratch(s, *c, &s3, &gm)) || (rc = adj_scratch(s, *c, &t7, &m3, &q))) return rc;
  if (has_inner(*c) && (rc = fat7_inner_dev(geo, *c, u, fs, s3, gm))) return rc;
  if (same) {
    if ((rc = fat7_adj_dev(geo, *c, u, fs, m, fs, lmid, fs, naik, s3, gm, t7, m3, q, d, fs, true))) return rc;
  } else {
    if ((rc = fat7_adj_dev(geo, *c, u, fs, m, fs, nullptr, 0, 0.0, s3, gm, t7, m3, q, d, fs, true))) return rc;
    if (want_long) {
      // the Naik term alone: a level with every fat7 coefficient zero
      qexstag_fat7_coefs z;
      std::memset(&z, 0, sizeof z);
      void *ptmp;
      if ((rc = s->ws.get(kSdTmp, field4_bytes(geo), &ptmp))) return rc;
      QS_CUDA(cudaMemsetAsync(ptmp, 0, field4_bytes(geo), stream()));
      if ((rc = fat7_adj_dev(geo, z, ul, fs, (const double2 *)ptmp, fs, lmid, fs, naik, nullptr, nullptr, nullptr,
                             nullptr, nullptr, dl, fs, true)))
        return rc;
    }
  }
  if ((rc = smear_out_finish(s, d, deriv, mem))) return rc;
  if (want_long && !same && (rc = smear_out_finish(s, dl, llderiv, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_project_u_deriv(qexstag_smear *s, const double *u, const double *x, const double *chain, double *r,
                            double eps, int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!u || !x || !chain || !r) return fail(QEXSTAG_ERR_ARG, "project_u_deriv: null argument");
  const double2 *du, *dx, *dc;
  double2 *dr;
  if ((rc = smear_in(s, kSmIn0, u, mem, &du)) || (rc = smear_in(s, kSmIn1, x, mem, &dx)) ||
      (rc = smear_in(s, kSdIn2, chain, mem, &dc)) || (rc = smear_out_buf(s, kSmOut0, r, mem, &dr)))
    return rc;
  if ((rc = project_u_deriv_dev(s->l->g, du, dx, dc, dr, eps)) || (rc = smear_out_finish(s, dr, r, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_hisq_deriv(qexstag_smear *s, const qexstag_hisq_coefs *c, const double *g, const double *cfat,
                       const double *clong, double *deriv, int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!c || !g || !cfat || !clong || !deriv) return fail(QEXSTAG_ERR_ARG, "hisq_deriv: null argument");
  if (!finite_coefs(c->fat7first) || !finite_coefs(c->fat7second) || !std::isfinite(c->naik))
    return fail(QEXSTAG_ERR_ARG, "hisq_deriv: coefficients not finite");
  const size_t fs = (size_t)9 * s->l->g.V;
  const double2 *u, *cf, *cl;
  double2 *d;
  if ((rc = smear_in(s, kSmIn0, g, mem, &u)) || (rc = smear_in(s, kSmIn1, cfat, mem, &cf)) ||
      (rc = smear_in(s, kSdIn2, clong, mem, &cl)) || (rc = smear_out_buf(s, kSmOut0, deriv, mem, &d)))
    return rc;
  if ((rc = hisq_deriv_dev(s, *c, u, cf, fs, cl, fs, d, false)) || (rc = smear_out_finish(s, d, deriv, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return QEXSTAG_OK;
}

int qexstag_hisq_force(qexstag_links *g, qexstag_smear *s, const qexstag_hisq_coefs *c, const double *thin,
                       double *f, const double *phi, double m, const qexstag_solver_params *p,
                       qexstag_solver_stats *st, int mem) {
  int rc;
  if ((rc = check_smear(s, mem))) return rc;
  if (!g || !g->u64 || !c || !thin || !f || !phi || !p) return fail(QEXSTAG_ERR_ARG, "hisq_force: null argument");
  if (g->nl != 8) return fail(QEXSTAG_ERR_ARG, "hisq_force: the link handle must hold 8 (fat+Naik) links");
  if (g->l != s->l) return fail(QEXSTAG_ERR_ARG, "hisq_force: handles on different layouts");
  if (!finite_coefs(c->fat7first) || !finite_coefs(c->fat7second) || !std::isfinite(c->naik))
    return fail(QEXSTAG_ERR_ARG, "hisq_force: coefficients not finite");
  const Geom &geo = s->l->g;
  const size_t fs = (size_t)9 * geo.V;
  const size_t vb = sizeof(double2) * 3 * (size_t)geo.V;
  const double2 *u, *dphi;
  double2 *df;
  void *ppsi, *pf8, *pff;
  if ((rc = smear_in(s, kSmIn0, thin, mem, &u)) || (rc = smear_out_buf(s, kSmOut0, f, mem, &df)) ||
      (rc = s->ws.get(kSfPsi, vb, &ppsi)) || (rc = s->ws.get(kSfF8, 2 * field4_bytes(geo), &pf8)) ||
      (rc = s->ws.get(kSfFF, field4_bytes(geo), &pff)))
    return rc;
  if (mem == QEXSTAG_MEM_DEVICE) {
    dphi = (const double2 *)phi;
  } else {
    void *soa, *aos;
    if ((rc = s->ws.get(kSfPhi, vb, &soa)) || (rc = s->ws.get(kSmAos, field4_bytes(geo) / 4, &aos))) return rc;
    QS_CUDA(cudaMemcpyAsync(aos, phi, vb, cudaMemcpyHostToDevice, stream()));
    if ((rc = aos_to_soa((const double *)aos, (double2 *)soa, geo.V, geo.V, 3))) return rc;
    dphi = (const double2 *)soa;
  }
  // smear the thin links into the operator (smearGetForce's forward part)
  if ((rc = hisq_dev(s, *c, u, g->u64, 2 * fs, g->u64 + fs, 2 * fs))) return rc;
  if ((rc = build_low_links(g))) return rc;
  // stagForceSolve, then fermForce's outer products f1 (fat) and f3 (long)
  double2 *psi = (double2 *)ppsi, *f8 = (double2 *)pf8, *ff = (double2 *)pff;
  const int status = qexstag_force_solve(g, (double *)psi, (const double *)dphi, m, p, st, QEXSTAG_MEM_DEVICE);
  if (status < 0) return status;
  if ((rc = qexstag_ferm_outer(g, (double *)f8, (const double *)psi, QEXSTAG_MEM_DEVICE))) return rc;
  // u.deriv(ff, f1, f3), then projectTAH(ff U^dag)
  if ((rc = hisq_deriv_dev(s, *c, u, f8, 2 * fs, f8 + fs, 2 * fs, ff, true))) return rc;
  tah_times_adj_kernel<<<field_grid(geo), kSmBlock, 0, stream()>>>(geo.V, ff, u, df, fs);
  note_launch();
  QS_LAUNCH_CHECK();
  if ((rc = smear_out_finish(s, df, f, mem))) return rc;
  QS_CUDA(cudaStreamSynchronize(stream()));
  return status;
}

}  // extern "C"
