// mrhs.cu -- QEX's multi-right-hand-side Dslash in FP64 (stagDN over
// stagDPN, src/physics/stagD.nim:132-189, 451-455): for n colour vectors at
// once, on one parity,
//   r_i = m x_i + sum_k [U_k(s) x_i(s + d_k) - U_k(s - d_k)^dagger x_i(s - d_k)].
// QEX tiles 16 sites x 8 vectors so that a site's links are loaded once for
// all vectors.  Here a block of 256 threads is G warp-uniform groups of
// 256/G sites (G = 1, 2 or 4); group q applies the operator to vectors
// 2q and 2q+1 of its sites.  Every group uses the same links, which come from
// HBM once per site: from L1 for the other groups, or through shared memory
// (the kernel with the ring, below).  Every vector's loads stay coalesced
// across the warp.  Up to 8 vectors per launch.  Accumulation follows stagDPN:
// the mass term, then the forward hops, then the backward hops.
//
// Compulsory bytes per output site: links (nlinks x 2 x 144 B: a forward
// link at the site and a backward link at the neighbour) + n x (48 B own
// site, 48 B neighbours (L2-resident), 48 B out) -> fat+Naik, n = 8:
// 2304 + 1152 = 3456 B, against 8 x 2448 B for eight single-vector sweeps.
#include <algorithm>

#include "lib.cuh"

namespace qs {

constexpr int kDnPer = 2;  // vectors per thread
constexpr int kDnMax = 8;  // vectors per launch

struct DnArgs {
  Geom g;
  const double2 *u;       // double2 [nlinks][9][V]
  int po;                 // output parity
  int n;                  // vectors in this launch
  int groups;             // G: threads of a block per site
  double m;
  const double2 *x[kDnMax];  // full-lattice fields, double2 [3][xstride]
  double2 *r[kDnMax];
  int xstride, rstride;
};

template <int NL>
__global__ void __launch_bounds__(kBlock, 2) dslashN64_kernel(const DnArgs A) {
  const Geom &g = A.g;
  const int nh = g.nh;
  const size_t V = (size_t)g.V;
  const int S = blockDim.x / A.groups;  // sites per block step
  const int grp = threadIdx.x / S, sl = threadIdx.x - grp * S;
  const int j0 = grp * kDnPer;
  if (j0 >= A.n) return;
  const int nq = min(kDnPer, A.n - j0);
  const size_t in_base = (size_t)(1 - A.po) * nh, out_base = (size_t)A.po * nh;
  for (int k = blockIdx.x * S + sl; k < nh; k += gridDim.x * S) {
    int x[4], lex;
    site_coords(g, A.po, k, x, lex);
    double2 acc[kDnPer][3];
#pragma unroll
    for (int q = 0; q < kDnPer; q++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        double2 v = make_double2(0.0, 0.0);
        if (q < nq) v = ldg(A.x[j0 + q] + (size_t)c * A.xstride + out_base + k);
        acc[q][c] = make_double2(A.m * v.x, A.m * v.y);
      }
    }
    // forward hops: + U_l(s) x(s + d_l)
#pragma unroll
    for (int l = 0; l < NL; l++) {
      const int mu = Hop<NL>::mu(l), len = Hop<NL>::len(l);
      const int jf = nbr_half(g, x, lex, mu, len);
      const double2 *ul = A.u + (size_t)l * 9 * V + out_base + k;
      double2 u[9];
#pragma unroll
      for (int e = 0; e < 9; e++) u[e] = ldlink(ul + (size_t)e * V);
#pragma unroll
      for (int q = 0; q < kDnPer; q++) {
        if (q < nq) {
          const double2 *xq = A.x[j0 + q] + in_base + jf;
          double2 v[3];
#pragma unroll
          for (int c = 0; c < 3; c++) v[c] = ldg(xq + (size_t)c * A.xstride);
#pragma unroll
          for (int i = 0; i < 3; i++)
#pragma unroll
            for (int c = 0; c < 3; c++) acc[q][i] = cmadd(acc[q][i], u[3 * i + c], v[c]);
        }
      }
    }
    // backward hops: - U_l(s - d_l)^dagger x(s - d_l)
#pragma unroll
    for (int l = 0; l < NL; l++) {
      const int mu = Hop<NL>::mu(l), len = Hop<NL>::len(l);
      const int jb = nbr_half(g, x, lex, mu, -len);
      const double2 *ul = A.u + (size_t)l * 9 * V + in_base + jb;
      double2 u[9];
#pragma unroll
      for (int e = 0; e < 9; e++) u[e] = ldlink(ul + (size_t)e * V);
#pragma unroll
      for (int q = 0; q < kDnPer; q++) {
        if (q < nq) {
          const double2 *xq = A.x[j0 + q] + in_base + jb;
          double2 w[3];
#pragma unroll
          for (int c = 0; c < 3; c++) w[c] = ldg(xq + (size_t)c * A.xstride);
#pragma unroll
          for (int i = 0; i < 3; i++) {
            double2 t = make_double2(0.0, 0.0);
#pragma unroll
            for (int c = 0; c < 3; c++) t = cjmadd(t, u[3 * c + i], w[c]);
            acc[q][i].x -= t.x;
            acc[q][i].y -= t.y;
          }
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kDnPer; q++) {
      if (q < nq) {
        double2 *rq = A.r[j0 + q] + out_base + k;
#pragma unroll
        for (int c = 0; c < 3; c++) rq[(size_t)c * A.rstride] = acc[q][c];
      }
    }
  }
}

// The same sums in the same order with more sites in flight.  The kernel above
// is bound by latency: its links and unrolled hops take the register file with
// 16 warps an SM.  Here the links of kDnAhead further terms are on their way to
// a ring in shared memory, which takes them out of the registers, and the terms
// run in a loop: 80 registers, 24 warps.  A block has one set of sites, and the
// blocks start in order, so that a hop's neighbours are still in L2 (six blocks
// an SM in strides over the sites: 340 us below).  24^3 x 48, fat+Naik, 8
// vectors: 388 -> 319 us, of 172 us for the compulsory bytes at 6.65 TB/s; what
// is left is the vectors' gathers.  The vectors in the ring as well took 360 us,
// their loads one term ahead in registers 382 us, the directions spread over
// warps 753 us.
template <int G>
constexpr int kDnAhead = G == 4 ? 3 : 1;  // what the 48 KB of a block hold

__device__ __forceinline__ void copy_link_async(double2 *dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

template <int NL, int G>
__global__ void __launch_bounds__(kBlock, 3) dslashN64_ring_kernel(const DnArgs A) {
  constexpr int S = kBlock / G;       // sites per block step
  constexpr int kTerms = 2 * NL;      // forward hops, then backward ones
  constexpr int kRing = kDnAhead<G> + 1;
  __shared__ double2 ring[kRing][9][S];
  const Geom &g = A.g;
  const int nh = g.nh;
  const size_t V = (size_t)g.V;
  const int grp = threadIdx.x / S, sl = threadIdx.x - grp * S;
  const int j0 = grp * kDnPer;
  const int nq = min(kDnPer, A.n - j0);  // may be <= 0: such a group copies links only
  const size_t in_base = (size_t)(1 - A.po) * nh, out_base = (size_t)A.po * nh;
  const int kk = blockIdx.x * S + sl, k = min(kk, nh - 1);
  int x[4], lex;
  site_coords(g, A.po, k, x, lex);
  auto nbr = [&](int n) {
    const int l = n < NL ? n : n - NL, len = Hop<NL>::len(l);
    return (lex + lex_step(g, x, Hop<NL>::mu(l), n < NL ? len : -len)) >> 1;
  };
  auto fetch = [&](int n) {
    if (n < kTerms) {
      const int l = n < NL ? n : n - NL;
      const double2 *ul = A.u + (size_t)l * 9 * V + (n < NL ? out_base + k : in_base + nbr(n));
#pragma unroll
      for (int e = 0; e < 9; e += G)
        if (e + grp < 9) copy_link_async(&ring[n % kRing][e + grp][sl], ul + (size_t)(e + grp) * V);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int n = 0; n < kDnAhead<G>; n++) fetch(n);
  double2 acc[kDnPer][3];
#pragma unroll
  for (int q = 0; q < kDnPer; q++) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      double2 v = make_double2(0.0, 0.0);
      if (q < nq) v = ldg(A.x[j0 + q] + (size_t)c * A.xstride + out_base + k);
      acc[q][c] = make_double2(A.m * v.x, A.m * v.y);
    }
  }
#pragma unroll 1
  for (int n = 0; n < kTerms; n++) {
    double2 v[kDnPer][3];
    const int jn = nbr(n);
#pragma unroll
    for (int q = 0; q < kDnPer; q++)
      if (q < nq) {
        const double2 *xq = A.x[j0 + q] + in_base + jn;
#pragma unroll
        for (int c = 0; c < 3; c++) v[q][c] = ldg(xq + (size_t)c * A.xstride);
      }
    asm volatile("cp.async.wait_group %0;" ::"n"(kDnAhead<G> - 1) : "memory");  // this thread's copies of term n
    __syncthreads();  // everyone's; and term n - 1's links have been read
    fetch(n + kDnAhead<G>);
    const int slot = n % kRing;
    if (n < NL) {  // forward: + U_l(s) x(s + d_l)
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double2 u = ring[slot][3 * i + c][sl];
#pragma unroll
          for (int q = 0; q < kDnPer; q++)
            if (q < nq) acc[q][i] = cmadd(acc[q][i], u, v[q][c]);
        }
    } else {  // backward: - U_l(s - d_l)^dagger x(s - d_l)
#pragma unroll
      for (int i = 0; i < 3; i++) {
        double2 t[kDnPer];
#pragma unroll
        for (int q = 0; q < kDnPer; q++) t[q] = make_double2(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double2 u = ring[slot][3 * c + i][sl];
#pragma unroll
          for (int q = 0; q < kDnPer; q++)
            if (q < nq) t[q] = cjmadd(t[q], u, v[q][c]);
        }
#pragma unroll
        for (int q = 0; q < kDnPer; q++) {
          acc[q][i].x -= t[q].x;
          acc[q][i].y -= t[q].y;
        }
      }
    }
  }
  if (kk < nh) {
#pragma unroll
    for (int q = 0; q < kDnPer; q++) {
      if (q < nq) {
        double2 *rq = A.r[j0 + q] + out_base + k;
#pragma unroll
        for (int c = 0; c < 3; c++) rq[(size_t)c * A.rstride] = acc[q][c];
      }
    }
  }
}

// The ring pays from about 260000 sites times vectors on for six and eight
// vectors, and from 490000 on for any more than two; below, its barriers cost more
// than its warps give.  In between an odd number leaves half of a group idle, and
// with three or four a block's 128 sites make a last wave that is nearly empty on
// some lattices (16^2 x 18 x 30: 540 blocks for 444 places).  us, first kernel / ring,
// fat+Naik, by sites times vectors in thousands: 3 vectors 207 38 / 46, 288 53 / 60,
// 498 97 / 89; 4 276 46 / 48, 327 62 / 56, 384 66 / 63, 664 112 / 97; 5 346 62 / 68, 480
// 94 / 91, 829 196 / 161; 6 295 56 / 54, 415 75 / 70, 576 114 / 93; 7 344 50 / 56, 484 73 /
// 72, 672 118 / 96; 8 262 43.7 / 42.9, 393 62 / 58, 553 83 / 75; naive 3 288 30 / 35, 498
// 53 / 52; 4 276 27 / 29, 384 36.9 / 37.6, 664 64 / 56; 5 408 43 / 46, 829 101 / 79; 6 295
// 31.7 / 31.6; 7 484 41.7 / 42.3, 672 68 / 55; 8 262 25 / 25, 393 35 / 34.  32^4 fat+Naik 3
// vectors 432 / 301, 8 663 / 553; 24^3 x 48 8 422 / 336.  One group, two vectors at most,
// has no use for it: 32^4 190 / 313.
constexpr long kDnRingFromFull = 262144, kDnRingFrom = 490000;

template <int NL>
static void launch_dn(const DnArgs &A) {
  const long nh = A.g.nh;
  const int S = kBlock / A.groups;
  const int sets = (int)((nh + S - 1) / S);
  const long from = A.n == 6 || A.n == 8 ? kDnRingFromFull : kDnRingFrom;
  if (A.groups == 1 || nh * A.n <= from)
    dslashN64_kernel<NL><<<std::min(sets, num_sms() * 4), kBlock, 0, stream()>>>(A);
  else if (A.groups == 2)
    dslashN64_ring_kernel<NL, 2><<<sets, kBlock, 0, stream()>>>(A);
  else
    dslashN64_ring_kernel<NL, 4><<<sets, kBlock, 0, stream()>>>(A);
}

// r[i] (parity po) = m x[i] + (2D) x[i] for i < n; full-lattice device
// fields with strides xstride, rstride.  Vectors go 8 to a launch.
int dslashN64(const qexstag_links_s *gl, int po, int n, double2 *const *r, int rstride, const double2 *const *x,
              int xstride, double m) {
  const Geom &g = gl->l->g;
  for (int i0 = 0; i0 < n; i0 += kDnMax) {
    DnArgs A;
    A.g = g;
    A.u = gl->u64;
    A.po = po;
    A.n = std::min(kDnMax, n - i0);
    A.groups = A.n <= 2 ? 1 : (A.n <= 4 ? 2 : 4);
    A.m = m;
    for (int j = 0; j < kDnMax; j++) {
      A.x[j] = j < A.n ? x[i0 + j] : nullptr;
      A.r[j] = j < A.n ? r[i0 + j] : nullptr;
    }
    A.xstride = xstride;
    A.rstride = rstride;
    if (gl->nl == 8)
      launch_dn<8>(A);
    else
      launch_dn<4>(A);
    note_launch();
    QS_LAUNCH_CHECK();
  }
  return QEXSTAG_OK;
}

}  // namespace qs
