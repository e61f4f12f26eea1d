// multishift.cu -- multi-shift CG (src/solvers/cgm.nim:68-246, after
// Jegerlehner, hep-lat/9612014) for several right-hand sides at once, and
// the drivers built on it:
//   solve_multishift: QEX's multi-mass solve (stagSolve.nim:560-668), FP64,
//     one right-hand side, every shift updated every iteration as cgm.nim does;
//   cgm_ee: (A + sigma_k) y_jk = b_j for up to 8 right-hand sides, with an
//     FP32 multi-right-hand-side Dslash that reads each link once per site for
//     all of them, shifts dropped once their residual |zeta_k| |r| meets the
//     target, then FP64 true residuals and, for every shift, a
//     multi-right-hand-side FP32 CG on the residuals of the right-hand sides
//     still above it (FP64 defect correction).
// All scalars (alpha, beta, zeta recurrences) live on the device in FP64.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "lib.cuh"
#include "lowprec.cuh"

namespace qs {

constexpr int kMaxShift = 32;
constexpr int kMaxRhs = 8;

struct CgmState {
  int itn, maxits, done, dropping;
  int nshift, nrhs;
  int last;           // the iteration that ended the last live right-hand side
  int pad0;
  int live[kMaxRhs];  // right-hand side still iterating
  double r2i[kMaxRhs], pAp[kMaxRhs], beta[kMaxRhs];
  double alphaim1[kMaxRhs], betaim1[kMaxRhs], r2stop[kMaxRhs], b2[kMaxRhs];
  double sg[kMaxShift];
  double zi[kMaxRhs][kMaxShift], zim1[kMaxRhs][kMaxShift];
  double cx[kMaxRhs][kMaxShift], cr[kMaxRhs][kMaxShift], cp[kMaxRhs][kMaxShift];
  int dox[kMaxRhs][kMaxShift], dop[kMaxRhs][kMaxShift], active[kMaxRhs][kMaxShift];
};

// Element types of the solve's vectors: double2 or float2, one right-hand
// side, or float4, a pair of them as (re_0, re_1, im_0, im_1), which one
// 16-byte load brings and one FP32x2 operation advances.
template <class VT>
struct Lanes {
  static constexpr int n = 1;
};
template <>
struct Lanes<float4> {
  static constexpr int n = 2;
};
__device__ __forceinline__ double2 &lane(double2 &v, int) { return v; }
__device__ __forceinline__ float2 &lane(float2 &v, int) { return v; }
struct Lane4 {
  float &x, &y;
};
__device__ __forceinline__ Lane4 lane(float4 &v, int q) { return q == 0 ? Lane4{v.x, v.z} : Lane4{v.y, v.w}; }

// vectors of the solve: [nrhs / n][3][nh] (r, Ap, t) and [nrhs / n][nshift][3][nh]
// (x, p), n right-hand sides to an element (an odd last one has a zero partner)
template <class VT>
struct CgmVecs {
  VT *r, *ap, *t, *x, *p;
  int nh, nshift, nvec;
  __host__ __device__ size_t rhs_off(int j) const { return (size_t)j * 3 * nh; }
  __host__ __device__ size_t xs_off(int j, int k) const { return ((size_t)j * nshift + k) * 3 * nh; }
};

// The sum over the grid of one double per right-hand side, from each warp's
// part: warps hold a part of right-hand side j in lane 0 and have stored it at
// partials[j * stride + slot]; the last block's warp j adds them in slot order
// of its lanes.  True in the last block, where sum is the total of right-hand
// side (warp) in every lane of that warp.  stride slots, blocks of kBlock
// threads (kMaxRhs warps).
__device__ __forceinline__ bool rhs_reduce(int nrhs, const double *partials, int stride, unsigned *ticket,
                                           unsigned nblocks, double &sum) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == nblocks - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  double s = 0.0;
  if (w < nrhs)
    for (int i = l; i < stride; i += 32) s += __ldcg(partials + (size_t)w * stride + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  sum = s;
  if (threadIdx.x == 0) *ticket = 0u;
  return true;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// FP32 multi-right-hand-side Dslash on pairs of right-hand sides.  A block is
// G = 1, 2 or 4 pairs by S = kBlock / G sites, a thread one pair of one site:
// a 16-byte vector load brings both right-hand sides, and the sums run in
// FP32x2 arithmetic with the link's parts broadcast.  Every operand passes
// through shared memory by asynchronous copies: a stage holds one hop's links
// of the block's sites, which its pairs share, and each thread's own vectors,
// and the copies run two or three hops ahead, from one set of sites to the next
// without a break.
//
// Bound by the latency of the gathers through L2: with loads to registers, one
// hop of 256 sites an SM in flight, a sweep at 16^4 fat+Naik with 8 right-hand
// sides took 24 us (32 us with the sums), whether a thread walked all hops or
// the directions were spread over warps; staged, 17 and 25 us, and 18 us for the
// second since cgm_update1 adds its blocks' sums (a last block that added them
// took 7 us).  Not faster: 128-thread blocks with the terms in a loop (19 us),
// four blocks an SM with three stages (18 and 20 us), a grid that gives every
// block as many sets (19 and 20 us).
// ---------------------------------------------------------------------------

// red_partials is shared by two sums: <p, Ap> from its start, |r|^2 behind it,
// kCgmSums doubles each over the right-hand sides
constexpr int kCgmSums = kMaxRedBlocks * 4;

struct MrhsArgs {
  Geom g;
  int po, nr, npair;
  LoLinks L;
  const float4 *xin;  // [npair][3][nh]
  const float4 *xs;   // [npair][3][nh] same-site operand (INIT)
  float4 *out;        // [npair][3][nh]
  size_t irs, srs, ors;  // pair strides of xin, xs, out
  int nh;
  float b;
  const CgmState *st;
  double *partials;
  Progress progress;  // posted by this launch (the first half sweep)
};

template <int G>
struct MrhsStage {
  static constexpr int kSites = kBlock / G, kStages = G == 4 ? 4 : G == 2 ? 3 : 2;
  float4 link[5][kSites];  // 18 reals (the last two in the first half of [4]) or 12
  float4 vec[G][3][kSites];
};

__device__ __forceinline__ unsigned shared_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(shared_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(shared_addr(dst)), "l"(src) : "memory");
}

// (re, im) += (ar, ai) (vr, vi) for both right-hand sides of a pair, nai = -ai
__device__ __forceinline__ void pair_mac(float2 &re, float2 &im, float ar, float ai, float nai, float2 vr, float2 vi) {
  const float2 ar2 = make_float2(ar, ar), ai2 = make_float2(ai, ai), nai2 = make_float2(nai, nai);
  re = __ffma2_rn(ar2, vr, re);
  re = __ffma2_rn(nai2, vi, re);
  im = __ffma2_rn(ar2, vi, im);
  im = __ffma2_rn(ai2, vr, im);
}

template <int NL, int HOP, int INIT, int RED, int R12, int G>
__global__ void __launch_bounds__(kBlock, 3) dslash_mrhs_kernel(const MrhsArgs A) {
  constexpr int S = MrhsStage<G>::kSites, kStages = MrhsStage<G>::kStages;
  constexpr int kTerms = 2 * NL;  // term n: link n / 2, forward (even n) or backward
  extern __shared__ __align__(16) unsigned char shared_bytes[];
  MrhsStage<G> *stage = reinterpret_cast<MrhsStage<G> *>(shared_bytes);
  pdl_wait();
  post_progress(A.progress);
  if (A.st->done) return;
  const Geom &g = A.g;
  const int nh = g.nh;
  const size_t V = (size_t)g.V;
  const size_t in_base = (size_t)(1 - A.po) * nh;
  const size_t out_base = (size_t)A.po * nh;
  const int pair = threadIdx.x / S, sl = threadIdx.x - pair * S;
  const bool on = pair < A.npair;  // the other threads copy links only
  struct Site {
    int k, lex, x[4];
  } cur, nxt;
  auto at = [&](int k0, Site &s) {
    s.k = min(k0 + sl, nh - 1);
    site_coords(g, A.po, s.k, s.x, s.lex);
  };
  // term n of site s into a stage
  auto fetch = [&](const Site &s, int n, int slot) {
    const int l = n >> 1, mu = Hop<NL>::mu(l), len = Hop<NL>::len(l);
    const bool lng = NL == 8 && (l & 1);
    const int f = NL == 8 ? (l >> 1) : l;
    const int jn = nbr_half(g, s.x, s.lex, mu, (n & 1) ? -len : len);
    const size_t us = (n & 1) ? in_base + jn : out_base + s.k;
    MrhsStage<G> &st = stage[slot];
    const int words = lng && R12 ? 3 : 4;
    const float4 *c = (lng ? A.L.f32_long : A.L.f32_fat) + (size_t)f * words * V + us;
#pragma unroll
    for (int e = 0; e < words; e += G)
      if (e + pair < words) copy16_async(&st.link[e + pair][sl], c + (size_t)(e + pair) * V);
    if (words == 4 && pair == 0)
      copy8_async(&st.link[4][sl], (lng ? A.L.f32_long_tail : A.L.f32_fat_tail) + (size_t)f * V + us);
    if (on) {
      const float4 *xp = A.xin + (size_t)pair * A.irs + jn;
#pragma unroll
      for (int i = 0; i < 3; i++) copy16_async(&st.vec[pair][i][sl], xp + (size_t)i * nh);
    }
  };
  const int step = gridDim.x * S;
  int slot = 0;  // of the term being summed
  at(blockIdx.x * S, cur);
#pragma unroll
  for (int n = 0; n < kStages - 1; n++) {
    fetch(cur, n, n);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  double dot[2] = {0.0, 0.0};
  for (int k0 = blockIdx.x * S; k0 < nh; k0 += step) {
    const bool more = k0 + step < nh;
    if (more) at(k0 + step, nxt);
    float2 re[3], im[3];
#pragma unroll
    for (int c = 0; c < 3; c++) re[c] = im[c] = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 0; n < kTerms; n++) {
      const int l = n >> 1, mu = Hop<NL>::mu(l);
      const bool lng = NL == 8 && (l & 1);
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");  // this thread's copies of term n
      __syncthreads();  // everyone's; and the term before has been read
      {
        const int ahead = n + kStages - 1;
        int to = slot + kStages - 1;
        if (to >= kStages) to -= kStages;
        if (ahead < kTerms)
          fetch(cur, ahead, to);
        else if (more)
          fetch(nxt, ahead - kTerms, to);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      const MrhsStage<G> &st = stage[slot];
      if (++slot == kStages) slot = 0;
      if (on) {
        float2 u[9];
#pragma unroll
        for (int e = 0; e < (lng && R12 ? 3 : 4); e++) {
          const float4 q = st.link[e][sl];
          u[2 * e] = make_float2(q.x, q.y);
          u[2 * e + 1] = make_float2(q.z, q.w);
        }
        if (lng && R12)
          recon_row2(u, ((n & 1) ? long_sign_bck(g, cur.x, mu) : long_sign_fwd(g, cur.x, mu)) * A.L.long_rc);
        else
          u[8] = *reinterpret_cast<const float2 *>(&st.link[4][sl]);
        float4 v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = st.vec[pair][c][sl];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const float2 vr = make_float2(v[c].x, v[c].y), vi = make_float2(v[c].z, v[c].w);
            // forward + U_ic v_c; backward - conj(U_ci) v_c
            if ((n & 1) == 0)
              pair_mac(re[i], im[i], u[3 * i + c].x, u[3 * i + c].y, -u[3 * i + c].y, vr, vi);
            else
              pair_mac(re[i], im[i], -u[3 * c + i].x, u[3 * c + i].y, -u[3 * c + i].y, vr, vi);
          }
      }
    }
    if (on && k0 + sl < nh) {
      float d0 = 0.f, d1 = 0.f;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        float4 o = make_float4(re[c].x, re[c].y, im[c].x, im[c].y);
        if (HOP < 0) o = make_float4(-o.x, -o.y, -o.z, -o.w);
        if (INIT) {
          const float4 s = __ldcg(A.xs + (size_t)pair * A.srs + (size_t)c * nh + cur.k);
          o.x = fmaf(A.b, s.x, o.x);
          o.y = fmaf(A.b, s.y, o.y);
          o.z = fmaf(A.b, s.z, o.z);
          o.w = fmaf(A.b, s.w, o.w);
          if (RED) {
            d0 = fmaf(s.x, o.x, fmaf(s.z, o.z, d0));
            d1 = fmaf(s.y, o.y, fmaf(s.w, o.w, d1));
          }
        }
        A.out[(size_t)pair * A.ors + (size_t)c * nh + cur.k] = o;
      }
      if (RED) {
        dot[0] += (double)d0;
        dot[1] += (double)d1;
      }
    }
    cur = nxt;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (RED) {
    // <xs, out>: a slot per warp and right-hand side (a warp holds one pair),
    // which the update's blocks add
    const int stride = gridDim.x * (S / 32), slot_ = blockIdx.x * (S / 32) + sl / 32;
    dot[0] = warp_sum(dot[0]);
    dot[1] = warp_sum(dot[1]);
    if (on && (threadIdx.x & 31) == 0) {
      A.partials[(size_t)(2 * pair) * stride + slot_] = dot[0];
      if (2 * pair + 1 < A.nr) A.partials[(size_t)(2 * pair + 1) * stride + slot_] = dot[1];
    }
  }
}

template <int NL, int R12, int G>
static int mrhs_pair(MrhsArgs A, int par, const float4 *p, size_t prs, float4 *t, float4 *ap, float b4m2, int *np) {
  constexpr int S = MrhsStage<G>::kSites, bytes = (int)sizeof(MrhsStage<G>) * MrhsStage<G>::kStages;
  auto *first = dslash_mrhs_kernel<NL, 1, 0, 0, R12, G>;
  auto *second = dslash_mrhs_kernel<NL, -1, 1, 1, R12, G>;
  QS_CUDA(cudaFuncSetAttribute(first, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  QS_CUDA(cudaFuncSetAttribute(second, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  // one wave of three blocks per SM; kCgmSums / nr partials per right-hand side
  const int grid = std::min({(A.nh + S - 1) / S, num_sms() * 3, kCgmSums / A.nr / (S / 32)});
  *np = grid * (S / 32);
  const size_t vs = (size_t)3 * A.nh;
  A.po = 1 - par;
  A.xin = p;
  A.irs = prs;
  A.xs = nullptr;
  A.srs = 0;
  A.out = t;
  A.ors = vs;
  A.b = 0.f;
  launch_pdl2(first, dim3(grid), kBlock, bytes, A);
  A.progress = Progress();
  A.po = par;
  A.xin = t;
  A.irs = vs;
  A.xs = p;
  A.srs = prs;
  A.out = ap;
  A.ors = vs;
  A.b = b4m2;
  launch_pdl2(second, dim3(grid), kBlock, bytes, A);
  note_launch(2);
  QS_LAUNCH_CHECK();
  return QEXSTAG_OK;
}

template <int NL, int R12>
static int mrhs_pairs(const MrhsArgs &A, int par, const float4 *p, size_t prs, float4 *t, float4 *ap, float b4m2,
                      int *np) {
  if (A.npair == 1) return mrhs_pair<NL, R12, 1>(A, par, p, prs, t, ap, b4m2, np);
  if (A.npair == 2) return mrhs_pair<NL, R12, 2>(A, par, p, prs, t, ap, b4m2, np);
  return mrhs_pair<NL, R12, 4>(A, par, p, prs, t, ap, b4m2, np);
}

// pair j of p at p + j*prs; of t and ap at j*3*nh.  *np: partials of <p, Ap>
// that each right-hand side has in red_partials
static int schur_mrhs(const qexstag_links_s *g, int par, int nr, const float4 *p, size_t prs, float4 *t,
                      float4 *ap, double m2, CgmState *st, const Progress &progress, int *np) {
  const Geom &geo = g->l->g;
  MrhsArgs A;
  A.g = geo;
  A.nr = nr;
  A.npair = (nr + 1) / 2;
  A.L = lo_links(g->low, kF32);
  A.nh = geo.nh;
  A.st = st;
  A.partials = red_partials();
  A.progress = progress;
  const float b4 = (float)(4.0 * m2);
  if (g->nl == 4) return mrhs_pairs<4, 0>(A, par, p, prs, t, ap, b4, np);
  return g->low.recon12 ? mrhs_pairs<8, 1>(A, par, p, prs, t, ap, b4, np)
                        : mrhs_pairs<8, 0>(A, par, p, prs, t, ap, b4, np);
}

// ---------------------------------------------------------------------------
// CG-M iteration kernels (element type VT); block row y works on element y of
// the vectors, so that every right-hand side has its own threads
// ---------------------------------------------------------------------------

template <class L1, class L2>
__device__ __forceinline__ void axpy2(L1 &&y, double a, L2 &&x) {
  using R = std::remove_reference_t<decltype(y.x)>;
  y.x = fma((R)a, x.x, y.x);
  y.y = fma((R)a, x.y, y.y);
}

// cgm.nim:157-184 for shift 0: r -= alpha Ap; x0 += alpha p0; |r|^2; then, in
// the last block, the zeta recurrences of every other shift (cgm.nim:187-200):
// warp j, lane k for shift k of right-hand side j.  alpha = r2 / <p, Ap>: with
// np > 0 every block adds the np partials that the operator left for its own
// right-hand sides at pap.  (One thread that walked the 8 x 6 scalars
// one by one, and two one-thread kernels around it for alpha and the end
// test, took 25 us an iteration at 16^4; this takes 11.5.  Whole 8-system,
// 6-shift solve: 238 -> 181 ms.)
template <class VT>
__global__ void __launch_bounds__(kBlock) cgm_update1_kernel(CgmVecs<VT> v, CgmState *st, const double *pap, int np,
                                                            double *partials, unsigned *ticket) {
  pdl_wait();
  if (st->done) return;
  constexpr int n = Lanes<VT>::n;
  const int nh = v.nh, e = blockIdx.y;
  __shared__ double sh[n * 32], sh_pap[n];
  double a[n], s[n];
  bool any = false;
  if (np > 0) {
    double t[n];
#pragma unroll
    for (int q = 0; q < n; q++) {
      t[q] = 0.0;
      if (e * n + q < st->nrhs)
        for (int i = threadIdx.x; i < np; i += blockDim.x) t[q] += __ldcg(pap + (size_t)(e * n + q) * np + i);
    }
    block_sum<n>(t, sh);
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < n; q++) {
        sh_pap[q] = t[q];
        if (blockIdx.x == 0 && e * n + q < st->nrhs) st->pAp[e * n + q] = t[q];  // for the last block
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < n; q++) {
    const int j = e * n + q;
    const bool on = j < st->nrhs && st->live[j] != 0;
    const double pAp = !on ? 0.0 : np > 0 ? sh_pap[q] : st->pAp[j];
    a[q] = pAp != 0.0 ? st->r2i[j] / pAp : 0.0;
    s[q] = 0.0;
    any |= on;
  }
  if (any) {
    VT *r = v.r + v.rhs_off(e);
    const VT *ap = v.ap + v.rhs_off(e);
    VT *x0 = v.x + v.xs_off(e, 0);
    const VT *p0 = v.p + v.xs_off(e, 0);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
      VT rv[3], xv[3], av[3], pv[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const size_t o = (size_t)c * nh + i;
        rv[c] = r[o];
        av[c] = ap[o];
        xv[c] = x0[o];
        pv[c] = p0[o];
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const size_t o = (size_t)c * nh + i;
#pragma unroll
        for (int q = 0; q < n; q++) {
          axpy2(lane(rv[c], q), -a[q], lane(av[c], q));
          axpy2(lane(xv[c], q), a[q], lane(pv[c], q));
          s[q] += (double)lane(rv[c], q).x * lane(rv[c], q).x + (double)lane(rv[c], q).y * lane(rv[c], q).y;
        }
        r[o] = rv[c];
        x0[o] = xv[c];
      }
    }
  }
  block_sum<n>(s, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < n; q++)
      if (e * n + q < st->nrhs) partials[(size_t)(e * n + q) * gridDim.x + blockIdx.x] = s[q];
  }
  double r2ip1;
  const int nrhs = st->nrhs, nshift = st->nshift;
  if (!rhs_reduce(nrhs, partials, gridDim.x, ticket, gridDim.x * gridDim.y, r2ip1)) return;
  const int j = threadIdx.x >> 5, k = threadIdx.x & 31;
  const int itn = st->itn + 1;
  int cont = 0;
  if (j < nrhs) {
    const bool live = st->live[j] != 0;
    const double pAp = __ldcg(&st->pAp[j]), r2i = st->r2i[j];
    const double alpha = pAp != 0.0 ? r2i / pAp : 0.0;
    const double beta = r2i != 0.0 ? r2ip1 / r2i : 0.0;
    cont = live && itn < st->maxits && r2ip1 > st->r2stop[j];
    int dox = 0, dop = 0;
    if (live && k > 0 && k < nshift && st->active[j][k]) {
      const double zi = st->zi[j][k], zim1 = st->zim1[j][k], sg = st->sg[k];
      double zip1d = alpha * st->betaim1[j] * (zim1 - zi);
      zip1d += zim1 * st->alphaim1[j] * (1.0 + sg * alpha);
      const double zip1 = (zip1d != 0.0) ? zi * zim1 * st->alphaim1[j] / zip1d : 0.0;
      const double zr = (zi != 0.0) ? zip1 / zi : 0.0;
      st->cx[j][k] = alpha * zr;
      dox = 1;
      if (cont) {
        dop = 1;
        st->cr[j][k] = zip1;
        st->cp[j][k] = beta * zr * zr;
        st->zim1[j][k] = zi;
        st->zi[j][k] = zip1;
        // the shifted residual is zeta_k r: stop updating a shift that meets it
        if (st->dropping && zip1 * zip1 * r2ip1 <= st->r2stop[j]) st->active[j][k] = 0;
      }
    }
    if (k < nshift) {
      st->dox[j][k] = dox;
      st->dop[j][k] = k == 0 ? cont : dop;
    }
    __syncwarp();
    if (k == 0 && live) {
      st->beta[j] = beta;
      st->alphaim1[j] = alpha;
      st->betaim1[j] = beta;
      st->r2i[j] = r2ip1;
      st->live[j] = cont;
    }
  }
  const int more = __syncthreads_or(cont);
  if (threadIdx.x == 0) {
    st->itn = itn;
    if (!more) {
      st->last = itn;
      st->done = 1;
    }
  }
}

// p0 = r + beta p0; x_k += cx p_k; p_k = cr r + cp p_k, of iteration it (the
// last one included: its x_k still move when update1 has ended the solve)
template <class VT>
__global__ void __launch_bounds__(kBlock) cgm_update2_kernel(CgmVecs<VT> v, const CgmState *st, int it) {
  pdl_wait();
  if (st->done && it > st->last) return;
  constexpr int n = Lanes<VT>::n;
  const int nh = v.nh, e = blockIdx.y, nshift = v.nshift;
  __shared__ double cx[n][kMaxShift], cr[n][kMaxShift], cp[n][kMaxShift];
  __shared__ int moves[kMaxShift], turns[n][kMaxShift];
  for (int t = threadIdx.x; t < nshift; t += blockDim.x) {
    int mv = 0;
#pragma unroll
    for (int q = 0; q < n; q++) {
      const int j = e * n + q;
      const bool on = j < st->nrhs;
      const int dox = on ? st->dox[j][t] : 0, dop = on ? st->dop[j][t] : 0;
      cx[q][t] = dox ? st->cx[j][t] : 0.0;
      cr[q][t] = t == 0 ? 1.0 : dop ? st->cr[j][t] : 0.0;
      cp[q][t] = dop ? (t == 0 ? st->beta[j] : st->cp[j][t]) : 0.0;
      turns[q][t] = dop;
      mv |= dox | dop;
    }
    moves[t] = mv;
  }
  __syncthreads();
  const VT *r = v.r + v.rhs_off(e);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
    VT rv[3];
#pragma unroll
    for (int c = 0; c < 3; c++) rv[c] = r[(size_t)c * nh + i];
    for (int k = 0; k < nshift; k++) {
      if (!moves[k]) continue;
      VT *xk = v.x + v.xs_off(e, k);
      VT *pk = v.p + v.xs_off(e, k);
      VT pv[3], xv[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        pv[c] = pk[(size_t)c * nh + i];
        if (k > 0) xv[c] = xk[(size_t)c * nh + i];
      }
#pragma unroll
      for (int c = 0; c < 3; c++) {
#pragma unroll
        for (int q = 0; q < n; q++) {
          if (k > 0) axpy2(lane(xv[c], q), cx[q][k], lane(pv[c], q));
          if (turns[q][k]) {
            VT z = rv[c];
            lane(z, q).x = 0;
            lane(z, q).y = 0;
            axpy2(lane(z, q), cr[q][k], lane(rv[c], q));
            axpy2(lane(z, q), cp[q][k], lane(pv[c], q));
            lane(pv[c], q).x = lane(z, q).x;
            lane(pv[c], q).y = lane(z, q).y;
          }
        }
        if (k > 0) xk[(size_t)c * nh + i] = xv[c];
        pk[(size_t)c * nh + i] = pv[c];
      }
    }
  }
}

// initial state: r = b, x = 0, p_k = r; |b|^2 per right-hand side
template <class VT>
__global__ void __launch_bounds__(kBlock) cgm_init_kernel(CgmVecs<VT> v, const double2 *const *b, int bstride,
                                                         CgmState *st, double *partials, unsigned *ticket,
                                                         double r2req) {
  constexpr int n = Lanes<VT>::n;
  const int nh = v.nh, e = blockIdx.y, nrhs = st->nrhs;
  __shared__ double sh[n * 32];
  double s[n];
#pragma unroll
  for (int q = 0; q < n; q++) s[q] = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x) {
    for (int c = 0; c < 3; c++) {
      VT rv{}, z{};
#pragma unroll
      for (int q = 0; q < n; q++) {
        const int j = e * n + q;
        if (j < nrhs) {
          const double2 bv = b[j][(size_t)c * bstride + i];
          lane(rv, q).x = bv.x;
          lane(rv, q).y = bv.y;
          s[q] += bv.x * bv.x + bv.y * bv.y;
        }
      }
      v.r[v.rhs_off(e) + (size_t)c * nh + i] = rv;
      for (int k = 0; k < v.nshift; k++) {
        v.x[v.xs_off(e, k) + (size_t)c * nh + i] = z;
        v.p[v.xs_off(e, k) + (size_t)c * nh + i] = rv;
      }
    }
  }
  block_sum<n>(s, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < n; q++)
      if (e * n + q < nrhs) partials[(size_t)(e * n + q) * gridDim.x + blockIdx.x] = s[q];
  }
  double tot;
  if (!rhs_reduce(nrhs, partials, gridDim.x, ticket, gridDim.x * gridDim.y, tot)) return;
  const int j = threadIdx.x >> 5, k = threadIdx.x & 31;
  int c = 0;
  if (j < nrhs) {
    c = (tot > r2req * tot) && isfinite(tot) ? 1 : 0;
    if (k == 0) {
      st->b2[j] = tot;
      st->r2i[j] = tot;
      st->r2stop[j] = r2req * tot;
      st->alphaim1[j] = -1.0;
      st->betaim1[j] = 0.0;
      st->live[j] = c;
    }
    if (k < st->nshift) {
      st->zi[j][k] = st->zim1[j][k] = 1.0;
      st->active[j][k] = 1;
      st->dox[j][k] = st->dop[j][k] = 0;
    }
  }
  const int any = __syncthreads_or(c);
  if (threadIdx.x == 0) {
    st->itn = 0;
    st->last = 0;
    st->done = (any && st->maxits > 0) ? 0 : 1;
  }
}

// right-hand side q of a vector's elements -> FP64 block of a full-lattice field
template <class VT>
__global__ void cgm_out_kernel(const VT *x, int q, int nh, double2 *y, int ystride, double scale) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nh; i += gridDim.x * blockDim.x)
    for (int c = 0; c < 3; c++) {
      VT v = x[(size_t)c * nh + i];
      y[(size_t)c * ystride + i] = make_double2(scale * (double)lane(v, q).x, scale * (double)lane(v, q).y);
    }
}

static int read_cgm_head(const CgmState *d, CgmState *h) {
  double *buf = host_results();
  const size_t n = offsetof(CgmState, r2i);
  QS_CUDA(cudaMemcpyAsync(buf, d, n, cudaMemcpyDeviceToHost, stream()));
  QS_CUDA(cudaStreamSynchronize(stream()));
  std::memcpy(h, buf, n);
  return QEXSTAG_OK;
}

int schur_lo_v32(const qexstag_links_s *g, int prec, int par, float2 *ap, const float2 *p, float2 *t, double m2,
                 double *dot_out, const Progress &progress);
int cg_mixed(qexstag_links_s *g, int par, double m2, CVecD b, VecD x, double r2req, int maxits, int sloppy,
             double delta, CgOut *out, int *reliable);

// Multi-shift CG on parity par: (A + sg[k]) x_jk = b_j, A = stagD2xx(m2),
// sg[0] = 0.  fp32: FP32 vectors with the multi-rhs FP32 Dslash (one
// right-hand side: the single-vector sloppy Schur with links of precision
// lprec, kF32 or kF16), else FP64 (nrhs must be 1).  Solutions are written
// to y[j*nshift+k] (FP64 blocks of parity par with stride ystride) scaled by
// yscale.
static int cgm_core(qexstag_links_s *g, int par, double m2, int nshift, const double *sg, int nrhs,
                    const double2 *const *b, int bstride, double2 *const *y, int ystride, double yscale,
                    double r2req, int maxits, bool fp32, bool dropping, int *iters, int lprec = kF32) {
  const Geom &geo = g->l->g;
  const int nh = geo.nh;
  Workspace &ws = g->ws;
  const bool pairs = fp32 && nrhs > 1;
  const int nvec = pairs ? (nrhs + 1) / 2 : nrhs;
  const size_t es = pairs ? sizeof(float4) : fp32 ? sizeof(float2) : sizeof(double2);
  const size_t vb = es * 3 * (size_t)nh;
  void *pr, *pap, *pt, *px, *pp, *pst, *pb;
  int rc;
  if ((rc = ws.get(kSlotMs0 + 40, vb * nvec, &pr)) || (rc = ws.get(kSlotMs0 + 41, vb * nvec, &pap)) ||
      (rc = ws.get(kSlotMs0 + 42, vb * nvec, &pt)) || (rc = ws.get(kSlotMs0 + 43, vb * nvec * nshift, &px)) ||
      (rc = ws.get(kSlotMs0 + 44, vb * nvec * nshift, &pp)) ||
      (rc = ws.get(kSlotMs0 + 45, sizeof(CgmState), &pst)) ||
      (rc = ws.get(kSlotMs0 + 46, sizeof(double2 *) * kMaxRhs, &pb)))
    return rc;
  CgmState *st = (CgmState *)pst;
  CgmState hs;
  std::memset(&hs, 0, sizeof(hs));
  hs.maxits = maxits;
  hs.nshift = nshift;
  hs.nrhs = nrhs;
  hs.dropping = dropping ? 1 : 0;
  for (int k = 0; k < nshift; k++) hs.sg[k] = (k == 0) ? 0.0 : sg[k];
  std::vector<char> staging(sizeof(CgmState) + sizeof(double2 *) * kMaxRhs);
  void *pin;
  if ((rc = ws.get_pinned(staging.size(), &pin))) return rc;
  std::memcpy(pin, &hs, sizeof(hs));
  std::memcpy((char *)pin + sizeof(hs), b, sizeof(double2 *) * nrhs);
  QS_CUDA(cudaMemcpyAsync(st, pin, sizeof(hs), cudaMemcpyHostToDevice, stream()));
  QS_CUDA(cudaMemcpyAsync(pb, (char *)pin + sizeof(hs), sizeof(double2 *) * nrhs, cudaMemcpyHostToDevice,
                          stream()));
  // grid rows share the GPU; kCgmSums / kMaxRhs slots per right-hand side
  const dim3 grid(std::min(grid_for(nh, kBlock, std::max(1, 8 / nvec)), kCgmSums / kMaxRhs), nvec);
  Pace pace;
  if ((rc = pace.start(ws, nh))) return rc;
  Progress progress;
  progress.word = pace.word;
  progress.itn = &st->itn;
  progress.stop = &st->done;
  int np = 0;  // <p, Ap> partials of the pair operator; the others finish the sum
  // an iteration: the operator's two half sweeps and the two updates
  auto solve = [&](auto v, auto schur) -> int {
    using VT = std::remove_pointer_t<decltype(v.r)>;
    cgm_init_kernel<VT><<<grid, kBlock, 0, stream()>>>(v, (const double2 *const *)pb, bstride, st, red_partials(),
                                                       red_tickets(), r2req);
    note_launch();
    QS_LAUNCH_CHECK();
    int rc2;
    for (;;) {
      unsigned long long seen;
      if ((rc2 = pace.wait(&seen))) return rc2;
      if (seen & kPaceStop) break;
      if ((rc2 = schur(v))) return rc2;
      pace.queued++;
      launch_pdl2(cgm_update1_kernel<VT>, grid, kBlock, 0, v, st, (const double *)red_partials(), np,
                  red_partials() + kCgmSums, red_tickets());
      launch_pdl2(cgm_update2_kernel<VT>, grid, kBlock, 0, v, (const CgmState *)st, (int)pace.queued);
      note_launch(2);
      QS_LAUNCH_CHECK();
    }
    if ((rc2 = read_cgm_head(st, &hs))) return rc2;
    constexpr int n = Lanes<VT>::n;
    const int egrid = grid_for(nh, kBlock, 8);
    for (int j = 0; j < nrhs; j++)
      for (int k = 0; k < nshift; k++) {
        cgm_out_kernel<VT><<<egrid, kBlock, 0, stream()>>>(v.x + v.xs_off(j / n, k), j % n, nh, y[j * nshift + k],
                                                           ystride, yscale);
        note_launch();
      }
    return QEXSTAG_OK;
  };
  if (pairs) {
    CgmVecs<float4> v{(float4 *)pr, (float4 *)pap, (float4 *)pt, (float4 *)px, (float4 *)pp, nh, nshift, nvec};
    // p_0 of pair j lives at xs_off(j, 0)
    rc = solve(v, [&](auto &w) {
      return schur_mrhs(g, par, nrhs, w.p, w.xs_off(1, 0), w.t, w.ap, m2, st, progress, &np);
    });
  } else if (fp32) {
    CgmVecs<float2> v{(float2 *)pr, (float2 *)pap, (float2 *)pt, (float2 *)px, (float2 *)pp, nh, nshift, 1};
    rc = solve(v, [&](auto &w) { return schur_lo_v32(g, lprec, par, w.ap, w.p, w.t, m2, &st->pAp[0], progress); });
  } else {
    if (nrhs != 1) return fail(QEXSTAG_ERR_ARG, "FP64 multi-shift takes one right-hand side");
    CgmVecs<double2> v{(double2 *)pr, (double2 *)pap, (double2 *)pt, (double2 *)px, (double2 *)pp, nh, nshift, 1};
    rc = solve(v, [&](auto &w) {
      return schur64(g, par, VecD{w.ap, nh}, CVecD{w.p, nh}, VecD{w.t, nh}, m2, kRedDot, nullptr, &st->done,
                     &st->pAp[0], progress);
    });
  }
  if (rc) return rc;
  QS_LAUNCH_CHECK();
  *iters = hs.itn;
  return QEXSTAG_OK;
}

int apply_D(qexstag_links_s *g, double2 *r, const double2 *x, double m, double sc);

// QEX's multi-mass solve (stagSolve.nim:560-668)
int solve_multishift(qexstag_links_s *g, int nmass, double2 *const *xs, const double2 *b,
                     const double *ms, const qexstag_solver_params *p, qexstag_solver_stats *st) {
  if (nmass > kMaxShift) return fail(QEXSTAG_ERR_ARG, "solve_multishift: at most 32 masses");
  const Geom &geo = g->l->g;
  const int V = geo.V, nh = geo.nh;
  Workspace &ws = g->ws;
  void *pr, *pxt;
  const size_t fb = sizeof(double2) * 3 * (size_t)V;
  int rc;
  if ((rc = ws.get(kSlotFull0, fb, &pr)) || (rc = ws.get(kSlotFull1, fb, &pxt))) return rc;
  double2 *r = (double2 *)pr, *xt = (double2 *)pxt;
  const double mass = ms[0];
  double b2e = 0, b2o = 0;
  if ((rc = vnorm2(block(b, geo, 0), nh, &b2e)) || (rc = vnorm2(block(b, geo, 1), nh, &b2o))) return rc;
  const double b2 = b2e + b2o;
  if (!std::isfinite(b2)) return fail(QEXSTAG_ERR_NAN, "solve_multishift: source is not finite");
  double r2 = b2;
  const double r2stop = p->r2req * b2;
  std::vector<double> shifts(nmass);
  for (int k = 0; k < nmass; k++) shifts[k] = (k == 0) ? 0.0 : 4.0 * (ms[k] * ms[k] - mass * mass);
  if ((rc = vcopy(VecD{r, V}, CVecD{b, V}, V)) || (rc = vzero(VecD{xt, V}, V))) return rc;
  for (int k = 0; k < nmass; k++)
    if ((rc = vzero(VecD{xs[k], V}, V))) return rc;
  const int maxits = p->maxits > 0 ? p->maxits : 50000;
  while (r2 > r2stop) {
    int mx = maxits - st->iterations;
    if (mx <= 0) break;
    double req = r2stop, r2s2 = 0.5 * req;
    double rse = (b2o <= r2s2) ? req - b2o : r2s2;
    double rso = (b2e <= r2s2) ? req - b2e : r2s2;
    int par;
    if (b2e > rse) {
      req = rse / b2e;
      par = 0;
    } else if (b2o > rso) {
      req = rso / b2o;
      par = 1;
    } else {
      break;
    }
    // cgm on parity par with r as the source; x_k[par] += 4 y_k
    std::vector<double2 *> ys(nmass);
    for (int k = 0; k < nmass; k++) {
      void *q;
      if ((rc = ws.get(kSlotMs0 + 60 + k, sizeof(double2) * 3 * (size_t)nh, &q))) return rc;
      ys[k] = (double2 *)q;
    }
    const double2 *rb = r + (size_t)par * nh;
    int its = 0;
    if ((rc = cgm_core(g, par, mass * mass, nmass, shifts.data(), 1, &rb, V, ys.data(), nh, 1.0, req, mx, false,
                       false, &its)))
      return rc;
    st->iterations += its;
    st->outer_iterations += 1;
    for (int k = 0; k < nmass; k++)
      if ((rc = vaxpy(block(xs[k], geo, par), 4.0, CVecD{ys[k], nh}, nh))) return rc;
    if ((rc = apply_D(g, xt, xs[0], mass, -1.0)) || (rc = apply_D(g, r, xt, mass, 1.0))) return rc;
    if ((rc = vsub(VecD{r, V}, CVecD{b, V}, CVecD{r, V}, V))) return rc;
    if ((rc = vnorm2(block((const double2 *)r, geo, 0), nh, &b2e)) ||
        (rc = vnorm2(block((const double2 *)r, geo, 1), nh, &b2o)))
      return rc;
    r2 = b2e + b2o;
    if (std::isnan(r2)) return fail(QEXSTAG_ERR_NAN, "solve_multishift: NaN residual");
  }
  // xs[k] = Ddag(ms[k]) xs[k]; for k = 0 that is xt from the last pass
  for (int k = 0; k < nmass; k++) {
    if (k != 0 && (rc = apply_D(g, xt, xs[k], ms[k], -1.0))) return rc;
    if ((rc = vcopy(VecD{xs[k], V}, CVecD{xt, V}, V))) return rc;
  }
  st->r2 = b2 > 0 ? r2 / b2 : 0.0;
  return (r2 > r2stop) ? QEXSTAG_NOT_CONVERGED : QEXSTAG_OK;
}

int cg64(qexstag_links_s *g, int par, double m2, CVecD b, VecD x, double r2req, int maxits, CgOut *out);

// (A + sigma) y on even sites, FP64: r = b - (A + sigma) y, returns |r|^2
static int shifted_residual(qexstag_links_s *g, double m2s, const double2 *bfull, const double2 *y, double2 *r,
                            double2 *t, double *r2) {
  const Geom &geo = g->l->g;
  const int nh = geo.nh;
  int rc;
  if ((rc = schur64(g, 0, VecD{r, nh}, block(y, geo, 0), VecD{t, nh}, m2s))) return rc;
  if ((rc = vsub(VecD{r, nh}, block(bfull, geo, 0), CVecD{r, nh}, nh))) return rc;
  return vnorm2(CVecD{r, nh}, nh, r2);
}

// even: no odd number of right-hand sides above one at a time
static int cgm_ee_run(qexstag_links_s *g, double m, int nshift, const double *sigma, int nrhs, const double2 *const *b,
                      double2 *const *y, const qexstag_solver_params *p, qexstag_solver_stats *st, double *r2_out,
                      bool even) {
  const Geom &geo = g->l->g;
  const int V = geo.V, nh = geo.nh;
  if (nshift > kMaxShift) return fail(QEXSTAG_ERR_ARG, "cgm_ee: at most 32 shifts");
  // base system: the smallest shift; the others relative to it
  int k0 = 0;
  for (int k = 1; k < nshift; k++)
    if (sigma[k] < sigma[k0]) k0 = k;
  std::vector<int> order(nshift);
  order[0] = k0;
  for (int k = 0, n = 1; k < nshift; k++)
    if (k != k0) order[n++] = k;
  std::vector<double> sg(nshift);
  for (int k = 0; k < nshift; k++) sg[k] = sigma[order[k]] - sigma[k0];
  const double m2 = m * m + 0.25 * sigma[k0];
  const int maxits = p->maxits > 0 ? p->maxits : 50000;
  const bool sloppy = p->sloppy != QEXSTAG_SLOPPY_NONE;
  // (a failed update of the links leaves older copies, or none)
  if (sloppy && !g->low.ready) return fail(QEXSTAG_ERR_STATE, "reduced-precision links missing");
  int rc;
  // zero the odd halves of the outputs
  for (int i = 0; i < nrhs * nshift; i++)
    if ((rc = vzero(block(y[i], geo, 1), nh))) return rc;
  // multi-shift phase, in batches of up to 8 right-hand sides
  const double r2ms = sloppy ? std::max(p->r2req, 1e-12) : p->r2req;
  for (int j0 = 0, nr; j0 < nrhs; j0 += nr) {
    nr = std::min(kMaxRhs, nrhs - j0);
    if (even && nr > 1) nr &= ~1;
    const double2 *bb[kMaxRhs];
    double2 *yy[kMaxRhs * kMaxShift];
    for (int j = 0; j < nr; j++) {
      bb[j] = b[j0 + j];
      for (int k = 0; k < nshift; k++) yy[j * nshift + k] = y[(j0 + j) * nshift + order[k]];
    }
    int its = 0;
    if (sloppy) {
      // FP32 links for the multi-shift phase at either sloppy precision: the
      // shifted solutions come out as accurate as the links they were
      // iterated with (about 1e-7 relative with FP32 links, 1e-4 with 16-bit
      // ones), and the per-shift refinement below, in the call's precision,
      // then covers three decades instead of six
      rc = cgm_core(g, 0, m2, nshift, sg.data(), nr, bb, V, yy, V, 1.0, r2ms, maxits, true, true, &its, kF32);
    } else {
      rc = 0;
      for (int j = 0; j < nr && !rc; j++) {
        int it1 = 0;
        rc = cgm_core(g, 0, m2, nshift, sg.data(), 1, &bb[j], V, &yy[j * nshift], V, 1.0, r2ms, maxits, false,
                      true, &it1);
        its += it1;
      }
    }
    if (rc) return rc;
    st->iterations += its;
  }
  st->outer_iterations += 1;
  // FP64 true residuals; refine every (j, k) above the target
  const size_t vb = sizeof(double2) * 3 * (size_t)nh;
  std::vector<double> b2(nrhs);
  for (int j = 0; j < nrhs; j++) {
    if ((rc = vnorm2(block(b[j], geo, 0), nh, &b2[j]))) return rc;
    if (!std::isfinite(b2[j])) return fail(QEXSTAG_ERR_NAN, "cgm_ee: source is not finite");
  }
  int status = QEXSTAG_OK;
  double worst = 0.0;
  if (sloppy) {
    // the right-hand sides of one shift together: a multi-right-hand-side
    // FP32 CG (cgm_core with the one shift) on their FP64 residuals, y += d,
    // repeated while any is above its target
    std::vector<double2 *> rbuf(kMaxRhs), dbuf(kMaxRhs);
    void *pt;
    for (int j = 0; j < kMaxRhs; j++) {
      void *a, *c;
      if ((rc = g->ws.get(kSlotMs0 + 100 + j, vb, &a)) || (rc = g->ws.get(kSlotMs0 + 110 + j, vb, &c))) return rc;
      rbuf[j] = (double2 *)a;
      dbuf[j] = (double2 *)c;
    }
    if ((rc = g->ws.get(kSlotMs0 + 51, vb, &pt))) return rc;
    double2 *t = (double2 *)pt;
    const double zero = 0.0;
    for (int k = 0; k < nshift; k++) {
      const double m2s = m * m + 0.25 * sigma[k];
      for (int j0 = 0; j0 < nrhs; j0 += kMaxRhs) {
        const int nr = std::min(kMaxRhs, nrhs - j0);
        std::vector<double> r2(nr);
        for (int j = 0; j < nr; j++)
          if ((rc = shifted_residual(g, m2s, b[j0 + j], y[(j0 + j) * nshift + k], rbuf[j], t, &r2[j]))) return rc;
        for (int pass = 0; pass < (even ? 20 : 10) && st->iterations < maxits; pass++) {
          // systems still above target, packed to the front
          std::vector<int> live;
          double req = 1.0;
          for (int j = 0; j < nr; j++) {
            const double stop = p->r2req * b2[j0 + j];
            if (r2[j] > stop) {
              live.push_back(j);
              req = std::min(req, 0.5 * stop / r2[j]);
            }
          }
          if (live.empty()) break;
          if (even && live.size() > 1 && live.size() % 2) live.pop_back();  // its turn comes in another pass
          req = std::max(req, 1e-12);  // what an FP32 inner solve can reach
          const double2 *rb[kMaxRhs];
          double2 *dy[kMaxRhs];
          for (size_t q = 0; q < live.size(); q++) {
            rb[q] = rbuf[live[q]];
            dy[q] = dbuf[live[q]];
          }
          int its = 0;
          if (live.size() == 1) {
            // one system: the reliable-update CG in the call's sloppy precision
            CgOut o{};
            int rel = 0;
            const double delta = p->delta > 0 ? p->delta : 0.1;
            if ((rc = cg_mixed(g, 0, m2s, CVecD{rb[0], nh}, VecD{dy[0], nh}, req, maxits - st->iterations,
                               p->sloppy, delta, &o, &rel)))
              return rc;
            its = o.iterations;
            st->reliable_updates += rel;
          } else if ((rc = cgm_core(g, 0, m2s, 1, &zero, (int)live.size(), rb, nh, dy, nh, 1.0, req,
                                    maxits - st->iterations, true, false, &its))) {
            return rc;
          }
          st->iterations += its;
          st->outer_iterations += 1;
          for (size_t q = 0; q < live.size(); q++) {
            const int j = live[q];
            double2 *yk = y[(j0 + j) * nshift + k];
            if ((rc = vaxpy(block(yk, geo, 0), 1.0, CVecD{dbuf[j], nh}, nh)) ||
                (rc = shifted_residual(g, m2s, b[j0 + j], yk, rbuf[j], t, &r2[j])))
              return rc;
          }
        }
        for (int j = 0; j < nr; j++) {
          const double rel2 = b2[j0 + j] > 0 ? r2[j] / b2[j0 + j] : 0.0;
          if (r2_out) r2_out[(j0 + j) * nshift + k] = rel2;
          worst = std::max(worst, rel2);
          if (r2[j] > p->r2req * b2[j0 + j]) status = QEXSTAG_NOT_CONVERGED;
        }
      }
    }
  } else {
    void *pr, *pt, *pd;
    if ((rc = g->ws.get(kSlotMs0 + 50, vb, &pr)) || (rc = g->ws.get(kSlotMs0 + 51, vb, &pt)) ||
        (rc = g->ws.get(kSlotMs0 + 52, vb, &pd)))
      return rc;
    double2 *r = (double2 *)pr, *t = (double2 *)pt, *d = (double2 *)pd;
    for (int j = 0; j < nrhs; j++) {
      for (int k = 0; k < nshift; k++) {
        const double m2s = m * m + 0.25 * sigma[k];
        double2 *yk = y[j * nshift + k];
        double r2 = 0;
        if ((rc = shifted_residual(g, m2s, b[j], yk, r, t, &r2))) return rc;
        const double r2stop = p->r2req * b2[j];
        int pass = 0;
        while (r2 > r2stop && pass < 10 && st->iterations < maxits) {
          CgOut o{};
          const int mx = maxits - st->iterations;
          if ((rc = cg64(g, 0, m2s, CVecD{r, nh}, VecD{d, nh}, 0.5 * r2stop / r2, mx, &o))) return rc;
          st->iterations += o.iterations;
          st->outer_iterations += 1;
          if ((rc = vaxpy(block(yk, geo, 0), 1.0, CVecD{d, nh}, nh))) return rc;
          if ((rc = shifted_residual(g, m2s, b[j], yk, r, t, &r2))) return rc;
          pass++;
        }
        const double rel2 = b2[j] > 0 ? r2 / b2[j] : 0.0;
        if (r2_out) r2_out[j * nshift + k] = rel2;
        worst = std::max(worst, rel2);
        if (r2 > r2stop) status = QEXSTAG_NOT_CONVERGED;
      }
    }
  }
  st->r2 = worst;
  return status;
}

int cgm_ee(qexstag_links_s *g, double m, int nshift, const double *sigma, int nrhs, const double2 *const *b,
           double2 *const *y, const qexstag_solver_params *p, qexstag_solver_stats *st, double *r2_out) {
  const qexstag_solver_stats start = *st;
  const int rc = cgm_ee_run(g, m, nshift, sigma, nrhs, b, y, p, st, r2_out, false);
  if (rc != QEXSTAG_ERR_ALLOC || p->sloppy == QEXSTAG_SLOPPY_NONE || nrhs % kMaxRhs == 1 || nrhs % 2 == 0) return rc;
  // memory is short, and the pair of an odd right-hand side is half empty:
  // once more with the odd one by itself
  for (int k = 40; k <= 44; k++) g->ws.drop(kSlotMs0 + k);
  *st = start;
  return cgm_ee_run(g, m, nshift, sigma, nrhs, b, y, p, st, r2_out, true);
}

}  // namespace qs
