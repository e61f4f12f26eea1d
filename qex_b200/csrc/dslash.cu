// dslash.cu -- FP64 even-odd staggered Dslash (naive and fat+Naik) and the
// Schur operator built from two half sweeps.
//
// One thread per output site.  For each hop k the thread gathers the input
// colour vector at s+d_k and s-d_k (other parity; neighbours of consecutive
// sites are nearly consecutive, so these gathers coalesce and the other-parity
// vector is served from L2 after its first read), streams the 9 complex
// elements of U_k(s) and of U_k(s-d_k) as 16-byte words, and accumulates
// U_k(s) x(s+d_k) - U_k(s-d_k)^dagger x(s-d_k) in registers (QEX stagD2,
// src/physics/stagD.nim:383-448: per k forward then backward, after the
// a*r + b*x init).  Neighbour indices come from the site coordinates
// (src/layout/qlayout.nim:108-136) rather than from tables, which saves
// 4 bytes per hop per site of HBM traffic.
//
// Compulsory HBM bytes per output site: 8 (naive) or 16 (fat+Naik) links of
// 144 B, plus 48 B in, 48 B out, plus 48 B per same-site init operand.
#include <algorithm>
#include <cstring>

#include "lib.cuh"

namespace qs {

struct DslashArgs64 {
  Geom g;
  int po;  // output parity; with both in one launch (BOTH) unused: even blocks work
           // on even sites, and the fields' pointers are those of the whole lattice
  const double2 *__restrict__ u;
  const double2 *__restrict__ xin;
  int istride;
  const double2 *xs;  // may alias out (same site, read before the write)
  int sstride;
  const double2 *rin;  // may alias out
  int rstride;
  double2 *out;
  int ostride;
  double a, b, c;
  const int *done;
  CgState *state;
  double *partials;
  unsigned *ticket;
  double *dot_out;
  // output sites: [k0, k0 + n1) then [k2, k2 + nsites - n1) of the parity
  // block (the whole block: k0 = k2 = 0, n1 = nsites = nh); with rowlen > 0
  // instead nsites / rowlen runs of rowlen sites, pitch apart, from k0
  int k0, n1, k2, nsites;
  int rowlen, pitch;
  Progress progress;  // posted by this launch (one of an iteration's half sweeps)
  CgFused cg;         // fused CG (CG > 0)
};

// Start of a fused CG iteration, in every block: the sum of the previous
// iteration's |r|^2, QEX's loop test (cg.nim:174) and beta.  All blocks add
// the same partials in the same order; block 0 records.  What other blocks
// read is not written here: rz alternates between two fields, and a block
// that finds done already set leaves as it would have by its own test.
__device__ __forceinline__ bool cg_begin(const CgFused &F, double *beta) {
  __shared__ double sh[32], sh_beta;
  __shared__ int sh_go;
  CgState *st = F.st;
  const int par = F.it & 1;
  if (__syncthreads_or(st->done)) return false;  // one answer for the block: block 0 of this launch may be setting it
  double v[1] = {0.0};
  if (F.it > 0) {
    for (int i = threadIdx.x; i < F.nr2; i += blockDim.x) v[0] += __ldcg(F.r2part + i);
    block_sum<1>(v, sh);
  }
  if (threadIdx.x == 0) {
    const double r2 = F.it > 0 ? v[0] : st->b2;
    const bool bad = isnan(r2);
    const bool go = F.it == 0 || (!bad && F.it < st->maxits && r2 > st->r2stop);
    sh_go = go;
    sh_beta = F.it > 0 ? r2 / st->rzs[par] : 0.0;
    if (blockIdx.x == 0) {
      st->r2 = r2;
      st->itn = F.it;
      if (go) {
        st->beta = sh_beta;
        st->rzs[par ^ 1] = r2;
      } else {
        st->nan = bad;
        st->done = 1;
      }
    }
  }
  __syncthreads();
  *beta = sh_beta;
  return sh_go;
}

// j-th output site of the launch, as an index of the parity block
__device__ __forceinline__ int out_site(const DslashArgs64 &A, int j) {
  if (A.rowlen > 0) {
    const int q = j / A.rowlen;
    return A.k0 + q * A.pitch + (j - q * A.rowlen);
  }
  return j < A.n1 ? A.k0 + j : A.k2 + (j - A.n1);
}

// the sum over the grid of each thread's part of <p, Ap>
template <int RED>
__device__ __forceinline__ void reduce_pap(const DslashArgs64 &A, double dot) {
  double v[1] = {dot}, s[1];
  if (grid_reduce<1>(v, A.partials, A.ticket, s) && threadIdx.x == 0) {
    if (RED == kRedCgPAp) {
      // cg.nim:213-215: qLAp = <q, LAp>, alpha = rz/qLAp; itn counted at Ap
      CgState *st = A.state;
      st->pAp = s[0];
      st->alpha = st->rz / s[0];
      st->itn += 1;
    } else {
      *A.dot_out = s[0];
    }
  }
}

// RESIDENT blocks per SM.  Without that bound the compiler stops at 72 to 90
// registers and waits for each hop's loads before it starts the next hop's; with
// 128 (two blocks) or 255 (one) it has the loads of several hops in flight, which
// is worth more than the warps it costs.  us, 72-90 registers / 128 / 255: Schur
// fat+Naik 32^4 423 / 374 / 380, 24^4 146 / 121 / 121, 16^4 64 / 29 / 26.5; naive
// 32^4 224 / 190 / 196, 24^4 79 / 62 / 66; D fat+Naik 32^4 361 / 289 / 291, naive
// 208 / 141 / 145; an FP64 CG iteration at 32^4 fat+Naik 534 / 424 / 427, naive 286
// / 241 / 247.  At 32^4 fat+Naik a half sweep then reads its compulsory bytes, and
// no more, from HBM at 6.9 TB/s, above the copy rate.  A block for every 256 sites
// instead of six per SM: 379.
template <int NL, int HOP, int INIT, int RED, int BOTH, int RESIDENT>
__global__ void __launch_bounds__(kBlock, RESIDENT) dslash64_kernel(const DslashArgs64 A) {
  pdl_wait();
  post_progress(A.progress);
  if (A.done != nullptr && *A.done) return;
  const Geom &g = A.g;
  const int nh = g.nh;
  const size_t V = (size_t)g.V;
  const int po = BOTH ? (int)(blockIdx.x & 1) : A.po;
  const int block = BOTH ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, blocks = gridDim.x >> BOTH;
  const size_t in_base = (size_t)(1 - po) * nh;
  const size_t out_base = (size_t)po * nh;
  const size_t in_off = BOTH ? in_base : 0, out_off = BOTH ? out_base : 0;
  const double2 *__restrict__ xin = A.xin + in_off;
  double dot = 0.0;
  for (int j = block * blockDim.x + threadIdx.x; j < A.nsites; j += blocks * blockDim.x) {
    const int k = out_site(A, j);
    int x[4], lex;
    site_coords(g, po, k, x, lex);
    double2 acc[3];
    double2 xsv[3];
    if (INIT == 0) {
#pragma unroll
      for (int c = 0; c < 3; c++) acc[c] = make_double2(0.0, 0.0);
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        xsv[c] = __ldcg(A.xs + (size_t)c * A.sstride + out_off + k);
        acc[c] = make_double2(A.b * xsv[c].x, A.b * xsv[c].y);
      }
      if (INIT == 2) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
          double2 rv = __ldcg(A.rin + (size_t)c * A.rstride + out_off + k);
          acc[c].x = fma(A.a, rv.x, acc[c].x);
          acc[c].y = fma(A.a, rv.y, acc[c].y);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < NL; l++) {
      const int mu = Hop<NL>::mu(l), len = Hop<NL>::len(l);
      const int jf = nbr_half(g, x, lex, mu, len);
      const int jb = nbr_half(g, x, lex, mu, -len);
      const double2 *ul = A.u + (size_t)l * 9 * V;
      double2 v[3], w[3], uf[9], ub[9];
#pragma unroll
      for (int c = 0; c < 3; c++) v[c] = ldg(xin + (size_t)c * A.istride + jf);
#pragma unroll
      for (int e = 0; e < 9; e++) uf[e] = ldlink(ul + (size_t)e * V + out_base + k);
#pragma unroll
      for (int c = 0; c < 3; c++) w[c] = ldg(xin + (size_t)c * A.istride + jb);
#pragma unroll
      for (int e = 0; e < 9; e++) ub[e] = ldlink(ul + (size_t)e * V + in_base + jb);
      double2 t[3], q[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        t[i] = make_double2(0.0, 0.0);
        q[i] = make_double2(0.0, 0.0);
#pragma unroll
        for (int j = 0; j < 3; j++) {
          t[i] = cmadd(t[i], uf[3 * i + j], v[j]);
          q[i] = cjmadd(q[i], ub[3 * j + i], w[j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        if (HOP > 0) {
          acc[i].x += t[i].x;
          acc[i].y += t[i].y;
          acc[i].x -= q[i].x;
          acc[i].y -= q[i].y;
        } else {
          acc[i].x -= t[i].x;
          acc[i].y -= t[i].y;
          acc[i].x += q[i].x;
          acc[i].y += q[i].y;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double2 o = make_double2(A.c * acc[c].x, A.c * acc[c].y);
      A.out[(size_t)c * A.ostride + out_off + k] = o;
      if (RED != kRedNone) {
        // Re <xs, out>, xs is the same-site operand (p in CG's A p)
        dot = fma(xsv[c].x, o.x, dot);
        dot = fma(xsv[c].y, o.y, dot);
      }
    }
  }
  if (RED != kRedNone) reduce_pap<RED>(A, dot);
}

// The same half sweep with a site's hops spread over the eight warps of a
// block: 32 sites per block step, warp w forming one link's two products
// (fat+Naik) or one of them (naive) for all 32, through shared memory to the
// threads (colour, site) that add them.  The products and the order of their
// sum are those of dslash64_kernel, so the result is the same bit for bit.
//
// Where the whole-site kernel has too few blocks to fill the GPU, its time
// is one thread's walk through 8 or 16 rounds of loads; this form takes one or
// two rounds.  With the GPU full it loses to the meeting in shared memory.  The
// figures are at kSplitMax.  At most 128 registers, for the same reason as above
// (12 x 10 x 14 x 18 fat+Naik: 22.4 us without the bound, 15.4); the sweeps of
// the fused CG (CG > 0) are faster without it (12^4 18 us an iteration, 21.6).
constexpr int kSplitSites = 32;
constexpr int kSplitWarps = kBlock / 32;

// CG > 0: the sweeps of a fused CG iteration.  CG = 1, the first, forms its
// input r + beta p at the neighbours; CG = 2, the second, forms p at its own
// sites and leaves each block's part of <p, Ap>.
template <int NL, int HOP, int INIT, int RED, int CG = 0, int BOTH = 0>
__global__ void __launch_bounds__(kBlock, CG ? 0 : 2) dslash64_split_kernel(const DslashArgs64 A) {
  constexpr int kTerms = 2 * NL, kPer = kTerms / kSplitWarps;
  __shared__ double2 term[kTerms][3][kSplitSites];
  pdl_wait();
  double beta = 0.0;
  if (CG == 1) {
    if (!cg_begin(A.cg, &beta)) return;
  } else if (CG == 2) {
    post_progress(A.progress);
    if (A.cg.st->done) return;
    beta = A.cg.st->beta;
  } else {
    post_progress(A.progress);
    if (A.done != nullptr && *A.done) return;
  }
  const Geom &g = A.g;
  const int nh = g.nh;
  const size_t V = (size_t)g.V;
  const int po = BOTH ? (int)(blockIdx.x & 1) : A.po;
  const int block = BOTH ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, blocks = gridDim.x >> BOTH;
  const size_t in_base = (size_t)(1 - po) * nh;
  const size_t out_base = (size_t)po * nh;
  const size_t in_off = BOTH ? in_base : 0, out_off = BOTH ? out_base : 0;
  const double2 *__restrict__ xin = A.xin + in_off;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double dot = 0.0;
  auto gather = [&](int n, double2 v[3]) {
#pragma unroll
    for (int c = 0; c < 3; c++) v[c] = ldg(xin + (size_t)c * A.istride + n);
    if (CG == 1 && A.cg.it > 0) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double2 pv = ldg(A.cg.p + (size_t)c * nh + n);
        v[c] = make_double2(fma(beta, pv.x, v[c].x), fma(beta, pv.y, v[c].y));
      }
    }
  };
  for (int j0 = block * kSplitSites; j0 < A.nsites; j0 += blocks * kSplitSites) {
    const bool on = j0 + lane < A.nsites;
    const int k = out_site(A, on ? j0 + lane : j0);
    int x[4], lex;
    site_coords(g, po, k, x, lex);
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int n = w * kPer + q, l = n >> 1;  // term n: link l, forward (even n) or backward
      const int mu = NL == 8 ? (l >> 1) : l, len = (NL == 8 && (l & 1)) ? 3 : 1;
      const double2 *ul = A.u + (size_t)l * 9 * V;
      double2 v[3], m[9], t[3];
      if ((n & 1) == 0) {
        const int jf = (lex + lex_step(g, x, mu, len)) >> 1;
#pragma unroll
        for (int e = 0; e < 9; e++) m[e] = ldlink(ul + (size_t)e * V + out_base + k);
        gather(jf, v);
#pragma unroll
        for (int i = 0; i < 3; i++) {
          t[i] = make_double2(0.0, 0.0);
#pragma unroll
          for (int c = 0; c < 3; c++) t[i] = cmadd(t[i], m[3 * i + c], v[c]);
        }
      } else {
        const int jb = (lex + lex_step(g, x, mu, -len)) >> 1;
#pragma unroll
        for (int e = 0; e < 9; e++) m[e] = ldlink(ul + (size_t)e * V + in_base + jb);
        gather(jb, v);
#pragma unroll
        for (int i = 0; i < 3; i++) {
          t[i] = make_double2(0.0, 0.0);
#pragma unroll
          for (int c = 0; c < 3; c++) t[i] = cjmadd(t[i], m[3 * c + i], v[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; c++) term[n][c][lane] = t[c];
    }
    __syncthreads();
    if (w < 3 && on) {
      const int c = w;
      double2 acc = make_double2(0.0, 0.0), xsv = acc;
      if (INIT > 0) {
        xsv = __ldcg(A.xs + (size_t)c * A.sstride + out_off + k);
        if (CG == 2) {  // xs is r
          double2 *p = A.cg.p + (size_t)c * nh + k;
          if (A.cg.it > 0) {
            const double2 pv = __ldcg(p);
            xsv = make_double2(fma(beta, pv.x, xsv.x), fma(beta, pv.y, xsv.y));
          }
          *p = xsv;
        }
        acc = make_double2(A.b * xsv.x, A.b * xsv.y);
      }
      if (INIT == 2) {
        const double2 rv = __ldcg(A.rin + (size_t)c * A.rstride + out_off + k);
        acc.x = fma(A.a, rv.x, acc.x);
        acc.y = fma(A.a, rv.y, acc.y);
      }
#pragma unroll
      for (int n = 0; n < kTerms; n++) {
        const double2 t = term[n][c][lane];
        if ((HOP > 0) == ((n & 1) == 0)) {
          acc.x += t.x;
          acc.y += t.y;
        } else {
          acc.x -= t.x;
          acc.y -= t.y;
        }
      }
      const double2 o = make_double2(A.c * acc.x, A.c * acc.y);
      A.out[(size_t)c * A.ostride + out_off + k] = o;
      if (RED != kRedNone || CG == 2) {
        dot = fma(xsv.x, o.x, dot);
        dot = fma(xsv.y, o.y, dot);
      }
    }
    __syncthreads();
  }
  if (CG == 2) {
    __shared__ double sh[32];
    double v[1] = {dot};
    block_sum<1>(v, sh);
    if (threadIdx.x == 0) A.cg.pap[blockIdx.x] = v[0];
  } else if (RED != kRedNone) {
    reduce_pap<RED>(A, dot);
  }
}

// Sites per launch up to which a half sweep spreads each site over a block's
// warps; above, a thread has a whole site, with 255 registers while there is no
// more than one block for each SM and 128 beyond.  Between the last lattice
// measured faster and the first slower.  Schur us, split / 255 / 128 registers:
//   fat+Naik 12^4 12.4 / 16.1 / 21.0, 14^4 18.9 / 19.9 / 24.2, 12^3 x 32 27.7 /
//   23.8 / 27.0, 16^4 30.8 / 26.5 / 29.1, 16^3 x 24 43.0 / 42.9 / 36.6
//   naive 14^4 10.4 / 11.3 / 12.9, 12^3 x 32 12.5 / 12.9 / 14.6, 16^4 15.5 / 14.5 /
//   16.2, 16^3 x 24 21.9 / 25.1 / 20.9, 24^4 61.4 / 65.8 / 61.6
//   D, fat+Naik 8^3 x 16 6.0 / 7.0 / 9.1, 8^3 x 32 7.2 / 7.7 / 9.9, 10^2 x 12 x 14 7.6 /
//   7.9 / 10.2, 12^4 9.5 / 8.2 / 10.3, 16^4 25.5 / 18.0 / 14.5; naive the launch's 5.9
//   in all three up to 10^2 x 12 x 14, 12^4 6.3 / 6.0 / 5.9, 16^4 16.3 / 10.6 / 8.4
template <int NL, int BOTH>
constexpr int kSplitMax = BOTH ? 16384 : NL == 8 ? 23000 : 30000;

template <int NL, int HOP, int INIT, int RED, int BOTH = 0>
static void launch64(const DslashArgs64 &A) {
  constexpr int par = BOTH + 1;  // parities in the launch
  if (par * A.nsites <= kSplitMax<NL, BOTH>) {
    const int grid = std::min((A.nsites + kSplitSites - 1) / kSplitSites, num_sms() * 3 / par);
    launch_pdl(dslash64_split_kernel<NL, HOP, INIT, RED, 0, BOTH>, par * grid, kBlock, A);
  } else {
    const int grid = par * grid_for(A.nsites, kBlock, 6 / par);
    if (grid <= num_sms())
      launch_pdl(dslash64_kernel<NL, HOP, INIT, RED, BOTH, 1>, grid, kBlock, A);
    else
      launch_pdl(dslash64_kernel<NL, HOP, INIT, RED, BOTH, 2>, grid, kBlock, A);
  }
  note_launch();
}

template <int NL>
static void launch_both(const DslashArgs64 &A, int init) {
  if (init == 0)
    launch64<NL, 1, 0, kRedNone, 1>(A);
  else if (init == 1)
    launch64<NL, 1, 1, kRedNone, 1>(A);
  else
    launch64<NL, 1, 2, kRedNone, 1>(A);
}

template <int NL>
static int dispatch64(const DslashArgs64 &A, int hop, int init, int red) {
#define QS_D64(H, I, R)                                            \
  if (hop == H && init == I && red == R) {                         \
    launch64<NL, H, I, R>(A);                                \
    return QEXSTAG_OK;                                             \
  }
  QS_D64(1, 0, kRedNone)
  QS_D64(1, 1, kRedNone)
  QS_D64(1, 2, kRedNone)
  QS_D64(-1, 0, kRedNone)
  QS_D64(-1, 1, kRedNone)
  QS_D64(-1, 2, kRedNone)
  QS_D64(-1, 1, kRedCgPAp)
  QS_D64(-1, 1, kRedDot)
#undef QS_D64
  return fail(QEXSTAG_ERR_ARG, "dslash64: unsupported variant");
}

int dslash64(const qexstag_links_s *gl, int po, VecD out, CVecD xin, CVecD xs, CVecD rin,
             double a, double b, double c, int hop, int init, int red, void *state,
             const int *done, double *dot_out, const Progress &progress) {
  const Geom &g = gl->l->g;
  DslashArgs64 A;
  A.progress = progress;
  A.g = g;
  A.po = po;
  A.u = gl->u64;
  A.xin = xin.p;
  A.istride = xin.stride;
  A.xs = xs.p;
  A.sstride = xs.stride;
  A.rin = rin.p;
  A.rstride = rin.stride;
  A.out = out.p;
  A.ostride = out.stride;
  A.a = a;
  A.b = b;
  A.c = c;
  A.done = done;
  A.state = (CgState *)state;
  A.partials = red_partials();
  A.ticket = red_tickets();
  A.dot_out = dot_out;
  A.k0 = A.k2 = 0;
  A.n1 = A.nsites = g.nh;
  A.rowlen = A.pitch = 0;
  int rc = (gl->nl == 8) ? dispatch64<8>(A, hop, init, red) : dispatch64<4>(A, hop, init, red);
  if (rc) return rc;
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// Both half sweeps of the operator on whole-lattice fields (stride V) in one
// launch: out = c (a rin + b x + (2D) x).  They are independent, and a link
// that one reads as the forward link of its own site the other reads as the
// backward link of a site nearby: side by side, the second read finds it in
// L2, where one launch after the other had the links from HBM twice.  D, us,
// two launches / one: 12 x 10 x 14 x 18 fat+Naik 18.2 / 9.3, 24^4 120 / 73, 32^4
// 371 / 289 (three time slices of links, the reach of the long hops, are most
// of L2 there); naive 24^4 61 / 37, 32^4 199 / 141.
int dslash64_both(const qexstag_links_s *gl, double2 *out, const double2 *x, const double2 *rin, double a, double b,
                  double c, int init) {
  const Geom &g = gl->l->g;
  DslashArgs64 A = {};
  A.g = g;
  A.u = gl->u64;
  A.xin = A.xs = x;
  A.rin = rin;
  A.out = out;
  A.istride = A.sstride = A.rstride = A.ostride = g.V;
  A.a = a;
  A.b = b;
  A.c = c;
  A.n1 = A.nsites = g.nh;
  if (gl->nl == 8)
    launch_both<8>(A, init);
  else
    launch_both<4>(A, init);
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// One half sweep over the sites [k0, k1) and [k2, k3) of parity po (either
// range may be empty): out = b xs + c (2D) xin with hop sign hop, no
// reduction; skipped once *done is set.  Used for the halo-overlapped
// Schur operator of a domain, whose interior sweeps run while the ghost
// slices are in flight.
int dslash64_ranges(const qexstag_links_s *gl, int po, VecD out, CVecD xin, CVecD xs, double b, double c,
                    int hop, int k0, int k1, int k2, int k3, const int *done) {
  const Geom &g = gl->l->g;
  if (k0 < 0 || k1 < k0 || k2 < 0 || k3 < k2 || k1 > g.nh || k3 > g.nh)
    return fail(QEXSTAG_ERR_ARG, "dslash64_ranges: site range outside the parity block");
  DslashArgs64 A = {};
  A.g = g;
  A.po = po;
  A.u = gl->u64;
  A.xin = xin.p;
  A.istride = xin.stride;
  A.xs = xs.p;
  A.sstride = xs.stride;
  A.out = out.p;
  A.ostride = out.stride;
  A.b = b;
  A.c = c;
  A.done = done;
  A.k0 = k0;
  A.n1 = k1 - k0;
  A.k2 = k2;
  A.nsites = (k1 - k0) + (k3 - k2);
  if (A.nsites == 0) return QEXSTAG_OK;
  const int init = xs.p ? 1 : 0;
  const int rc = (gl->nl == 8) ? dispatch64<8>(A, hop, init, kRedNone) : dispatch64<4>(A, hop, init, kRedNone);
  if (rc) return rc;
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// One half sweep over nrun runs of rowlen sites of parity po, pitch apart,
// from k0 (a block of z rows in each of a range of t slices): out = b xs +
// c (2D) xin with hop sign hop, no reduction; skipped once *done is set.
int dslash64_rows(const qexstag_links_s *gl, int po, VecD out, CVecD xin, CVecD xs, double b, double c, int hop,
                  int k0, int nrun, int rowlen, int pitch, const int *done) {
  const Geom &g = gl->l->g;
  if (k0 < 0 || nrun < 0 || rowlen < 0 || rowlen > pitch ||
      (nrun > 0 && (long)k0 + (long)(nrun - 1) * pitch + rowlen > g.nh))
    return fail(QEXSTAG_ERR_ARG, "dslash64_rows: site runs outside the parity block");
  DslashArgs64 A = {};
  A.g = g;
  A.po = po;
  A.u = gl->u64;
  A.xin = xin.p;
  A.istride = xin.stride;
  A.xs = xs.p;
  A.sstride = xs.stride;
  A.out = out.p;
  A.ostride = out.stride;
  A.b = b;
  A.c = c;
  A.done = done;
  A.k0 = k0;
  A.rowlen = rowlen;
  A.pitch = pitch;
  A.nsites = nrun * rowlen;
  A.n1 = A.nsites;
  if (A.nsites == 0) return QEXSTAG_OK;
  const int init = xs.p ? 1 : 0;
  const int rc = (gl->nl == 8) ? dispatch64<8>(A, hop, init, kRedNone) : dispatch64<4>(A, hop, init, kRedNone);
  if (rc) return rc;
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// Whether an FP64 CG takes the fused iteration, whose sweeps are spread over
// warps: on small lattices, and where the whole-site form would have a second
// round of blocks (two on an SM) that is at most a third full.  Iteration us,
// fused / not: fat+Naik 12^3 x 32 30 / 34, 16^4 38 / 37, 16^2 x 18 x 30 64 / 60; by
// blocks for 296 places 297 72 / 80, 313 74 / 83, 325 75 / 84, 344 82 / 86, 366 87 / 89,
// 375 88 / 90, 384 87 / 90, 395 95 / 92, 432 100 / 97; naive 12^3 x 32 19.2 / 24.8, 16^3 x
// 14 21.5 / 25.6, 16^4 22.9 / 21.5, 270 blocks 40.9 / 38.0, 297 45.6 / 47.9, 325 47.2 /
// 50.5, 344 51.8 / 51.4, 375 54.2 / 53.7, 384 53.7 / 53.7, 395 57.4 / 54.5.
bool cg_fused_fits(const qexstag_links_s *gl) {
  const int nh = gl->l->g.nh, blocks = (nh + kBlock - 1) / kBlock, places = 2 * num_sms();
  return nh <= 30000 || (blocks > places && blocks <= places + places / 3);
}

// the two half sweeps of a fused CG iteration; *npap: the <p, Ap> partials
int schur64_fused(const qexstag_links_s *gl, int par, const CgFused &F, double m2, const Progress &progress, int *npap) {
  const Geom &g = gl->l->g;
  DslashArgs64 A = {};
  A.g = g;
  A.u = gl->u64;
  A.n1 = A.nsites = g.nh;
  A.cg = F;
  A.c = 1.0;
  const int grid = std::min((g.nh + kSplitSites - 1) / kSplitSites, num_sms() * 3);
  A.po = 1 - par;
  A.xin = F.r;
  A.istride = g.nh;
  A.out = F.t;
  A.ostride = g.nh;
  if (gl->nl == 8)
    launch_pdl(dslash64_split_kernel<8, 1, 0, kRedNone, 1>, grid, kBlock, A);
  else
    launch_pdl(dslash64_split_kernel<4, 1, 0, kRedNone, 1>, grid, kBlock, A);
  A.po = par;
  A.xin = F.t;
  A.xs = F.r;
  A.sstride = g.nh;
  A.out = F.ap;
  A.b = 4.0 * m2;
  A.progress = progress;  // its work covers the report's wait, the other kernels' is shorter
  if (gl->nl == 8)
    launch_pdl(dslash64_split_kernel<8, -1, 1, kRedNone, 2>, grid, kBlock, A);
  else
    launch_pdl(dslash64_split_kernel<4, -1, 1, kRedNone, 2>, grid, kBlock, A);
  note_launch(2);
  *npap = grid;
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

// stagD2xx (stagD.nim:485-512): t_q = (2D)_{q,par} x (stagDP, rir := 0), then
// r = 4 m2 x - (2D)_{par,q} t (stagDM with rir := 4 m2 x).
int schur64(const qexstag_links_s *gl, int par, VecD r, CVecD x, VecD t, double m2, int red,
            void *state, const int *done, double *dot_out, const Progress &progress) {
  int rc = dslash64(gl, 1 - par, t, x, CVecD{nullptr, 0}, CVecD{nullptr, 0}, 0.0, 0.0, 1.0, +1,
                    0, kRedNone, nullptr, done, nullptr, progress);
  if (rc) return rc;
  return dslash64(gl, par, r, cv(t), x, CVecD{nullptr, 0}, 0.0, 4.0 * m2, 1.0, -1, 1, red, state,
                  done, dot_out);
}

}  // namespace qs

namespace qs {

// The FP64 Schur operator with a caller-provided temporary t, launched
// without touching the library's reduction scratch (no reductions, no
// early exit); used by the allocation-free entry point.
int schur64_plain(const qexstag_links_s *gl, int par, VecD r, CVecD x, VecD t, double m2) {
  const Geom &g = gl->l->g;
  DslashArgs64 A = {};
  A.g = g;
  A.u = gl->u64;
  A.n1 = A.nsites = g.nh;
  // t = (2D)_{q,par} x
  A.po = 1 - par;
  A.xin = x.p;
  A.istride = x.stride;
  A.out = t.p;
  A.ostride = t.stride;
  A.c = 1.0;
  if (gl->nl == 8)
    launch64<8, 1, 0, kRedNone>(A);
  else
    launch64<4, 1, 0, kRedNone>(A);
  // r = 4 m2 x - (2D)_{par,q} t
  A.po = par;
  A.xin = t.p;
  A.istride = t.stride;
  A.xs = x.p;
  A.sstride = x.stride;
  A.out = r.p;
  A.ostride = r.stride;
  A.b = 4.0 * m2;
  if (gl->nl == 8)
    launch64<8, -1, 1, kRedNone>(A);
  else
    launch64<4, -1, 1, kRedNone>(A);
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

}  // namespace qs
