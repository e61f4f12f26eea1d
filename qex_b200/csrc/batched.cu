// batched.cu -- many independent even-odd CG solves in one persistent
// launch.
//
// Each problem j has its own lattice (own dims), links, mass and source and
// solves stagD2ee(m_j^2) x_j = b_j on its even sites with QEX's CG
// (src/solvers/cg.nim:174-240, cpNone).  Small lattices cannot fill a B200
// alone and a per-problem solve is bound by kernel launches; here every
// problem's sites, in sets of 32, are laid end to end, split into equal
// contiguous chunks, one per block of a cooperative grid (again whenever a
// problem ends, so that the last, slowest problems still use every SM), and
// the whole CG runs inside one kernel:
//   phase A  t_j = (2D)_oe p_j  with p_j = r_j + beta_j p_j formed at the
//            neighbours on the fly (odd output sites)
//   phase B  p_j = r_j + beta_j p_j; Ap_j = 4 m_j^2 p_j - (2D)_eo t_j; <p_j, Ap_j>
//   phase C  x_j += alpha_j p_j; r_j -= alpha_j Ap_j; |r_j|^2
// separated by grid barriers.  In the sweeps a set's hops are spread over the
// block's eight warps, which meet in shared memory (as in the one-lattice
// kernel for small lattices).  A block leaves one partial sum per problem of
// its chunk; after the barrier every block adds the partials that it needs in
// the same fixed order, so all take the same decisions without a further
// step, and results are bitwise reproducible.  Finished problems drop out; the
// kernel returns when none is active.  16 lattices of 2048 to 8192 even sites:
// 7.4 ms, where a thread per site, a ticket per problem with its last block
// finishing the sums, and a barrier of two hops took 10.9 ms; the links through
// L2, 150 MB an iteration while all are active, are 12 of its 31 us.
//
// Every wait is bounded: a barrier that has not completed within the time
// limit sets an error flag and all blocks return; the host reports
// QEXSTAG_ERR_TIMEOUT.  Data written inside the kernel is read with L2-only
// loads, because L1 is not coherent across SMs.
#include <algorithm>
#include <cstring>
#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

#include "batch_part.cuh"
#include "lib.cuh"

namespace qs {

int cg64(qexstag_links_s *g, int par, double m2, CVecD b, VecD x, double r2req, int maxits, CgOut *out);

constexpr int kBatchBlock = 256;
constexpr int kBatchWarps = kBatchBlock / 32;
constexpr int kSetSites = 32;

struct BProb {
  Geom g;
  const double2 *u;  // [nl][9][V]
  const double2 *b;  // even block of b (stride V)
  double2 *x;        // even block of x (stride V)
  double2 *r, *p, *ap, *t;  // [3][nh]
  double m2;
};

// the problem set, uploaded for every call
struct BSet {
  int nprob, maxits;
  double r2req;
  BProb prob[kMaxBatch];
};

struct BState {
  double r2, b2;
  int itn, pad;
};

struct BGlobal {
  unsigned arrived;  // blocks that have reached a barrier, over all barriers so far
  int err;
};

struct BArgs {
  const BSet *set;
  BState *st;
  BGlobal *glob;
  double *part;  // two arrays of part_stride partials: <p, Ap> and |r|^2
  int part_stride;
  long long timeout_cycles;
};

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------

__device__ __forceinline__ int ld_int(const int *p) { return *(volatile const int *)p; }
__device__ __forceinline__ double2 ld2(const double2 *p) { return __ldcg(p); }

// Grid barrier with a time limit; returns false (in every thread) when the
// barrier failed or another block reported an error.  Arrivals are counted
// without ever being reset, so the last one's own increment releases the
// others; target is the count this barrier waits for, kept by each block.
// missing > 0 makes the barrier wait for that many blocks that do not exist
// (the self-test's stand-in for a block that never arrives).
__device__ bool grid_sync(BGlobal *gl, unsigned &target, long long timeout, unsigned missing = 0) {
  __shared__ int ok;
  target += gridDim.x + missing;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned n;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(n) : "l"(&gl->arrived) : "memory");
    n += 1;
    ok = 1;
    const long long t0 = clock64();
    for (unsigned spins = 0; (int)(n - target) < 0; spins++) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&gl->arrived) : "memory");
      if ((spins & 31) == 31) {
        if (ld_int(&gl->err)) break;
        if (clock64() - t0 > timeout) {
          atomicExch(&gl->err, 1);
          break;
        }
      }
    }
    if (ld_int(&gl->err)) ok = 0;
    __threadfence();
  }
  __syncthreads();
  return ok;
}

// every block passes the barrier twice; out = 1 when both passed
__global__ void barrier_selftest_kernel(BGlobal *gl, long long timeout, unsigned missing, int *out) {
  unsigned target = 0;
  const bool a = grid_sync(gl, target, timeout, missing);
  const bool b = a && grid_sync(gl, target, timeout, missing);
  if (blockIdx.x == 0 && threadIdx.x == 0) *out = (a && b) ? 1 : 0;
}

template <int NL>
struct BShared {
  static constexpr int kBufs = NL == 4 ? 2 : 1;
  double2 term[kBufs][2 * NL][3][kSetSites];
  BProb prob[kMaxBatch];
  BPart T;
  double red[kBatchWarps][kMaxMet];
  double rz[kMaxBatch], stop[kMaxBatch], alpha[kMaxBatch], beta[kMaxBatch];
  int itn[kMaxBatch], done[kMaxBatch];
};

__device__ __forceinline__ int sets_of(int nh) { return (nh + kSetSites - 1) / kSetSites; }

// thread 0 builds the partition over the problems that are not done
template <int NL>
__device__ void build_part(BShared<NL> &S, int nprob) {
  __syncthreads();
  if (threadIdx.x == 0)
    fill_part(
        S.T, nprob, [&](int j) { return S.done[j]; }, [&](int j) { return sets_of(S.prob[j].g.nh); }, gridDim.x,
        blockIdx.x);
  __syncthreads();
}

// this block's sums of red over its warps, one per problem, to its slots:
// block b's part of active problem i lies at b + i
template <int NL>
__device__ __forceinline__ void leave_partials(BShared<NL> &S, double *part, int warps) {
  __syncthreads();
  for (int q = threadIdx.x; q < S.T.np; q += blockDim.x) {
    double v = 0.0;
    for (int w = 0; w < warps; w++) v += S.red[w][q];
    part[blockIdx.x + S.T.i0 + q] = v;
  }
}
// the sum of active problem i's partials, by one warp, in every lane
__device__ __forceinline__ double sum_partials(const BPart &T, const double *part, int i) {
  const int b0 = block_of(T, T.soff[i]), b1 = block_of(T, T.soff[i + 1] - 1);
  double v = 0.0;
  for (int b = b0 + (threadIdx.x & 31); b <= b1; b += 32) v += __ldcg(part + b + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// The hop sums of this block's sets on the output sites of parity po.  gather(Q,
// j, n, v) gives problem j's input vector at neighbour n; out(Q, j, k, c, sum)
// takes colour c of site k's sum of the hops, forward ones positive, in warps
// 0 to 2 (warp = c); leave(i) is called in those warps after the last set of
// the block's i-th problem.
template <int NL, class Gather, class Out, class Leave>
__device__ __forceinline__ void hop_sums(BShared<NL> &S, int po, Gather gather, Out out, Leave leave) {
  constexpr int kTerms = 2 * NL, kPer = kTerms / kBatchWarps;
  const BPart &T = S.T;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int i = T.i0, buf = 0;
  for (int s = T.s0; s < T.s1; s++) {
    while (s >= T.soff[i + 1]) i++;
    const int j = T.ids[i];
    const BProb &Q = S.prob[j];
    const Geom &g = Q.g;
    const size_t V = (size_t)g.V;
    const size_t in_base = (size_t)(1 - po) * g.nh, out_base = (size_t)po * g.nh;
    const int k0 = (s - T.soff[i]) * kSetSites + lane;
    const bool on = k0 < g.nh;
    const int k = on ? k0 : g.nh - 1;
    int x[4], lex;
    site_coords(g, po, k, x, lex);
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int n = w * kPer + q, l = n >> 1, back = n & 1;
      const int mu = NL == 8 ? (l >> 1) : l, len = (NL == 8 && (l & 1)) ? 3 : 1;
      const int jn = (lex + lex_step(g, x, mu, back ? -len : len)) >> 1;
      const double2 *ul = Q.u + (size_t)l * 9 * V + (back ? in_base + jn : out_base + k);
      double2 v[3], m[9], t[3];
#pragma unroll
      for (int e = 0; e < 9; e++) m[e] = ldg(ul + (size_t)e * V);
      gather(Q, j, jn, v);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        t[a] = make_double2(0.0, 0.0);
#pragma unroll
        for (int c = 0; c < 3; c++)
          t[a] = back ? cjmadd(t[a], m[3 * c + a], v[c]) : cmadd(t[a], m[3 * a + c], v[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; c++) S.term[buf][n][c][lane] = t[c];
    }
    __syncthreads();
    if (w < 3) {
      if (on) {
        double2 acc = make_double2(0.0, 0.0);
#pragma unroll
        for (int n = 0; n < kTerms; n += 2) {
          const double2 f = S.term[buf][n][w][lane], b = S.term[buf][n + 1][w][lane];
          acc.x += f.x - b.x;
          acc.y += f.y - b.y;
        }
        out(Q, j, k, w, acc);
      }
      if (s + 1 == T.s1 || s + 1 == T.soff[i + 1]) leave(i - T.i0);
    }
    // with two buffers the next set's terms go to the other one, and its own
    // meeting keeps the set after that away from this one
    if (BShared<NL>::kBufs == 2)
      buf ^= 1;
    else
      __syncthreads();
  }
}

// pointwise work on the block's even sites, a warp at a time on (set, colour);
// f(Q, j, k, c) returns the site's part of a sum, which is left in red
template <int NL, class F>
__device__ __forceinline__ void pointwise(BShared<NL> &S, F f) {
  const BPart &T = S.T;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q = threadIdx.x; q < kBatchWarps * T.np; q += blockDim.x) S.red[q / T.np][q % T.np] = 0.0;
  __syncthreads();
  int i = T.i0;
  double acc = 0.0;
  for (int t = w; t < 3 * (T.s1 - T.s0); t += kBatchWarps) {
    const int s = T.s0 + t / 3, c = t % 3;
    if (s >= T.soff[i + 1]) {
      acc = lanes_sum(acc);
      if (lane == 0) S.red[w][i - T.i0] = acc;
      acc = 0.0;
      while (s >= T.soff[i + 1]) i++;
    }
    const int j = T.ids[i];
    const BProb &Q = S.prob[j];
    const int k = (s - T.soff[i]) * kSetSites + lane;
    if (k < Q.g.nh) acc += f(Q, j, k, c);
  }
  acc = lanes_sum(acc);
  if (lane == 0 && T.np > 0) S.red[w][i - T.i0] = acc;
}

// Two blocks on an SM: with 108 registers a warp has its link's loads in flight
// together, where the 64 that the compiler takes without the bound (three blocks)
// make it wait in between (16 lattices, naive, 8 x 8 x 8 x 16 and its like: 7.99 ->
// 7.35 ms).
template <int NL>
__global__ void __launch_bounds__(kBatchBlock, 2) batched_cg_kernel(const BArgs A) {
  extern __shared__ __align__(16) unsigned char shared_bytes[];
  BShared<NL> &S = *reinterpret_cast<BShared<NL> *>(shared_bytes);
  const int nprob = A.set->nprob, maxits = A.set->maxits;
  const double r2req = A.set->r2req;
  const long long tmo = A.timeout_cycles;
  double *const pap = A.part, *const pr2 = A.part + A.part_stride;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned target = 0;
  for (int j = threadIdx.x; j < nprob; j += blockDim.x) {
    S.prob[j] = A.set->prob[j];
    S.done[j] = 0;
    S.itn[j] = 0;
    S.beta[j] = 0.0;
  }
  build_part(S, nprob);

  // ---- init: r = b, x = 0, p = 0; |b|^2 ----
  pointwise(S, [&](const BProb &Q, int, int k, int c) {
    const int V = Q.g.V, nh = Q.g.nh;
    const double2 bv = ldg(Q.b + (size_t)c * V + k);
    Q.r[(size_t)c * nh + k] = bv;
    Q.p[(size_t)c * nh + k] = make_double2(0.0, 0.0);
    Q.x[(size_t)c * V + k] = make_double2(0.0, 0.0);
    return fma(bv.x, bv.x, bv.y * bv.y);
  });
  leave_partials(S, pr2, kBatchWarps);
  if (!grid_sync(A.glob, target, tmo)) return;
  for (int i = w; i < S.T.na; i += kBatchWarps) {
    const double b2 = sum_partials(S.T, pr2, i);
    if (lane == 0) {
      const int j = S.T.ids[i];
      S.rz[j] = b2;
      S.stop[j] = r2req * b2;
      S.done[j] = (!(b2 > S.stop[j]) || maxits <= 0 || isnan(b2)) ? 1 : 0;
      if (blockIdx.x == 0) A.st[j] = BState{b2, b2, 0, 0};
    }
  }
  build_part(S, nprob);

  while (S.T.na > 0) {
    // ---- phase A: t = (2D)_oe (r + beta p) on odd sites ----
    hop_sums<NL>(
        S, 1,
        [&](const BProb &Q, int j, int n, double2 v[3]) {
          const int nh = Q.g.nh;
          const double beta = S.beta[j];
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double2 rv = ld2(Q.r + (size_t)c * nh + n), pv = ld2(Q.p + (size_t)c * nh + n);
            v[c] = make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
          }
        },
        [&](const BProb &Q, int, int k, int c, double2 sum) { Q.t[(size_t)c * Q.g.nh + k] = sum; }, [](int) {});
    if (!grid_sync(A.glob, target, tmo)) return;
    // ---- phase B: p = r + beta p; Ap = 4 m2 p - (2D)_eo t; <p, Ap> ----
    double dot = 0.0;
    hop_sums<NL>(
        S, 0,
        [&](const BProb &Q, int, int n, double2 v[3]) {
#pragma unroll
          for (int c = 0; c < 3; c++) v[c] = ld2(Q.t + (size_t)c * Q.g.nh + n);
        },
        [&](const BProb &Q, int j, int k, int c, double2 sum) {
          const size_t o = (size_t)c * Q.g.nh + k;
          const double2 rv = ld2(Q.r + o), po = ld2(Q.p + o);
          const double beta = S.beta[j];
          const double2 pv = make_double2(fma(beta, po.x, rv.x), fma(beta, po.y, rv.y));
          const double2 av = make_double2(4.0 * Q.m2 * pv.x - sum.x, 4.0 * Q.m2 * pv.y - sum.y);
          Q.p[o] = pv;
          Q.ap[o] = av;
          dot = fma(pv.x, av.x, dot);
          dot = fma(pv.y, av.y, dot);
        },
        [&](int q) {
          dot = lanes_sum(dot);
          if (lane == 0) S.red[w][q] = dot;
          dot = 0.0;
        });
    leave_partials(S, pap, 3);
    if (!grid_sync(A.glob, target, tmo)) return;
    for (int q = w; q < S.T.np; q += kBatchWarps) {
      const double s = sum_partials(S.T, pap, S.T.i0 + q);
      const int j = S.T.ids[S.T.i0 + q];
      if (lane == 0) S.alpha[j] = S.rz[j] / s;
    }
    __syncthreads();
    // ---- phase C: x += alpha p; r -= alpha Ap; |r|^2 ----
    pointwise(S, [&](const BProb &Q, int j, int k, int c) {
      const size_t o = (size_t)c * Q.g.nh + k, ox = (size_t)c * Q.g.V + k;
      const double alpha = S.alpha[j];
      const double2 pv = ld2(Q.p + o), av = ld2(Q.ap + o);
      double2 xv = ld2(Q.x + ox), rv = ld2(Q.r + o);
      xv.x = fma(alpha, pv.x, xv.x);
      xv.y = fma(alpha, pv.y, xv.y);
      rv.x = fma(-alpha, av.x, rv.x);
      rv.y = fma(-alpha, av.y, rv.y);
      Q.x[ox] = xv;
      Q.r[o] = rv;
      return fma(rv.x, rv.x, rv.y * rv.y);
    });
    leave_partials(S, pr2, kBatchWarps);
    if (!grid_sync(A.glob, target, tmo)) return;
    int ended = 0;
    for (int i = w; i < S.T.na; i += kBatchWarps) {
      const double r2 = sum_partials(S.T, pr2, i);
      const int j = S.T.ids[i];
      const int itn = S.itn[j] + 1;
      const int d = (!(itn < maxits && r2 > S.stop[j]) || isnan(r2)) ? 1 : 0;
      __syncwarp();
      if (lane == 0) {
        S.beta[j] = r2 / S.rz[j];
        S.rz[j] = r2;
        S.itn[j] = itn;
        S.done[j] = d;
        if (d && blockIdx.x == 0) {
          A.st[j].r2 = r2;
          A.st[j].itn = itn;
        }
      }
      ended |= d;
    }
    if (__syncthreads_or(ended)) build_part(S, nprob);
  }
}

// the barrier's state at the start of a solve (first node of the captured
// graph, so that a relaunch starts from scratch)
__global__ void batched_reset_kernel(BGlobal *gl) {
  gl->arrived = 0;
  gl->err = 0;
}

// ---------------------------------------------------------------------------
// host side: arena, launch configuration (autotuned), graph
// ---------------------------------------------------------------------------

namespace {

struct BatchCache {
  std::mutex m;  // one batch at a time on a device
  void *arena = nullptr;
  size_t bytes = 0;
  void *pinned = nullptr;  // BSet up, BGlobal and the states down
  cudaStream_t stream = nullptr;
  std::map<std::vector<long>, int> tuned;  // blocks per SM by (nl, sets)
  // The captured solve.  Its kernels find everything that differs from call to
  // call in the uploaded set, so it depends on these alone.
  int gnl = 0, gper_sm = 0;
  cudaGraphExec_t exec = nullptr;
};
BatchCache g_bc[64];

int cache_of(BatchCache **out) {
  int d = 0;
  cudaGetDevice(&d);
  if (d < 0 || d >= 64) return fail(QEXSTAG_ERR_ARG, "device out of range");
  *out = &g_bc[d];
  return QEXSTAG_OK;
}

// blocks of the solver per SM, 0 when it cannot run
template <int NL>
int max_blocks() {
  int n = 0;
  const int bytes = (int)sizeof(BShared<NL>);
  if (cudaFuncSetAttribute(batched_cg_kernel<NL>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batched_cg_kernel<NL>, kBatchBlock, bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

constexpr int kMaxPerSm = 8;

// the arena's fixed part
struct BArena {
  BSet set;
  BState st[kMaxBatch];
  BGlobal glob;
};

}  // namespace

// enqueue reset + the cooperative persistent kernel on s (capturable)
static int enqueue_batched(const BatchCache *bc, int nl, int per_sm, cudaStream_t s) {
  BArena *ar = (BArena *)bc->arena;
  BArgs A;
  A.set = &ar->set;
  A.st = ar->st;
  A.glob = &ar->glob;
  A.part = (double *)((char *)bc->arena + ((sizeof(BArena) + 255) & ~(size_t)255));
  A.part_stride = num_sms() * kMaxPerSm + kMaxBatch;
  A.timeout_cycles = 4000000000LL;  // ~2 s at the boost clock
  batched_reset_kernel<<<1, 1, 0, s>>>(A.glob);
  QS_LAUNCH_CHECK();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_sms() * per_sm);
  cfg.blockDim = dim3(kBatchBlock);
  cfg.dynamicSmemBytes = nl == 8 ? sizeof(BShared<8>) : sizeof(BShared<4>);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = nl == 8 ? cudaLaunchKernelEx(&cfg, batched_cg_kernel<8>, A)
                          : cudaLaunchKernelEx(&cfg, batched_cg_kernel<4>, A);
  if (e != cudaSuccess) return cuda_fail(e, "cooperative launch of batched_cg_kernel");
  return QEXSTAG_OK;
}

// The solve as a CUDA graph: [reset, persistent kernel], captured once per
// launch configuration and relaunched after that.  Returns 1 in *used when
// the graph ran, 0 when capture was refused and the kernels were launched
// directly instead.
static int graph_batched(BatchCache *bc, int nl, int per_sm, int *used) {
  cudaStream_t s = bc->stream;
  note_launch(2);
  if (!(bc->exec && bc->gnl == nl && bc->gper_sm == per_sm)) {
    if (bc->exec) cudaGraphExecDestroy(bc->exec);
    bc->exec = nullptr;
    cudaGraph_t graph = nullptr;
    int rc = QEXSTAG_OK;
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      rc = enqueue_batched(bc, nl, per_sm, s);
      e = cudaStreamEndCapture(s, &graph);
    }
    if (e == cudaSuccess && rc == QEXSTAG_OK && graph) e = cudaGraphInstantiate(&bc->exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess || rc != QEXSTAG_OK || !bc->exec) {
      cudaGetLastError();
      bc->exec = nullptr;
      *used = 0;
      return enqueue_batched(bc, nl, per_sm, s);
    }
    bc->gnl = nl;
    bc->gper_sm = per_sm;
  }
  QS_CUDA(cudaGraphLaunch(bc->exec, s));
  *used = 1;
  return QEXSTAG_OK;
}

// Upload the set with this limit on the iterations, run it, wait, and check
// the barrier's error flag; the states come back behind it.
static int run_batched(BatchCache *bc, int nl, int per_sm, int maxits, bool graph, int *used) {
  BArena *host = (BArena *)bc->pinned, *dev = (BArena *)bc->arena;
  host->set.maxits = maxits;
  const size_t up = offsetof(BSet, prob) + sizeof(BProb) * host->set.nprob;
  QS_CUDA(cudaMemcpyAsync(&dev->set, &host->set, up, cudaMemcpyHostToDevice, bc->stream));
  int rc = graph ? graph_batched(bc, nl, per_sm, used) : enqueue_batched(bc, nl, per_sm, bc->stream);
  if (rc) return rc;
  QS_CUDA(cudaMemcpyAsync(host->st, dev->st, sizeof(BArena) - offsetof(BArena, st), cudaMemcpyDeviceToHost,
                          bc->stream));
  QS_CUDA(cudaStreamSynchronize(bc->stream));
  if (host->glob.err) return fail(QEXSTAG_ERR_TIMEOUT, "batched solve: a grid barrier timed out");
  return QEXSTAG_OK;
}

// blocks per SM: each timed over a fixed number of iterations, the fastest kept
static int tune(BatchCache *bc, int nl, long nsets, int *per_sm) {
  std::vector<long> key{nl, nsets};
  auto it = bc->tuned.find(key);
  if (it != bc->tuned.end()) {
    *per_sm = it->second;
    return QEXSTAG_OK;
  }
  const int mx = std::min(nl == 8 ? max_blocks<8>() : max_blocks<4>(), kMaxPerSm);
  if (mx < 1) return fail(QEXSTAG_ERR_CUDA, "batched solve: the kernel does not fit an SM");
  double best = 1e30;
  int bp = 1;
  cudaEvent_t e0, e1;
  QS_CUDA(cudaEventCreate(&e0));
  QS_CUDA(cudaEventCreate(&e1));
  int rc = QEXSTAG_OK;
  for (int ps = 1; ps <= mx && !rc; ps++)
    for (int rep = 0; rep < 2 && !rc; rep++) {  // the first run of a shape pays for its launch
      cudaEventRecord(e0, bc->stream);
      rc = run_batched(bc, nl, ps, 12, false, nullptr);
      cudaEventRecord(e1, bc->stream);
      cudaEventSynchronize(e1);
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep && ms < best) {
        best = ms;
        bp = ps;
      }
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  bc->tuned[key] = bp;
  *per_sm = bp;
  return QEXSTAG_OK;
}

int solve_batched(int nprob, qexstag_links_s *const *gs, const double *mass, double2 *const *x,
                  const double2 *const *b, const qexstag_solver_params *p, int *iters, double *r2_out,
                  qexstag_solver_stats *st, int *tuned_block, int *tuned_per_sm, int *graph_used) {
  BatchCache *bc;
  int rc = cache_of(&bc);
  if (rc) return rc;
  std::lock_guard<std::mutex> lock(bc->m);
  if (!bc->stream) QS_CUDA(cudaStreamCreateWithFlags(&bc->stream, cudaStreamNonBlocking));
  if (!bc->pinned) QS_CUDA(cudaHostAlloc(&bc->pinned, sizeof(BArena), cudaHostAllocDefault));
  const int nl = gs[0]->nl;
  long nsets = 0;
  auto vec_bytes = [](int nh) { return (sizeof(double2) * 3 * (size_t)nh + 255) & ~(size_t)255; };
  const size_t fixed = ((sizeof(BArena) + 255) & ~(size_t)255) +
                       ((2 * sizeof(double) * ((size_t)num_sms() * kMaxPerSm + kMaxBatch) + 255) & ~(size_t)255);
  size_t bytes = fixed;
  for (int j = 0; j < nprob; j++) {
    const int nh = gs[j]->l->g.nh;
    bytes += 4 * vec_bytes(nh);
    nsets += (nh + kSetSites - 1) / kSetSites;
  }
  if (bc->bytes < bytes) {
    if (bc->arena) {
      cudaDeviceSynchronize();
      cudaFree(bc->arena);
      bc->arena = nullptr;
      bc->bytes = 0;
    }
    if (bc->exec) cudaGraphExecDestroy(bc->exec);
    bc->exec = nullptr;
    cudaError_t e = device_malloc(&bc->arena, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      bc->arena = nullptr;
      return fail(QEXSTAG_ERR_ALLOC, "batched solve: device allocation failed");
    }
    bc->bytes = bytes;
  }
  BArena *host = (BArena *)bc->pinned;
  host->set.nprob = nprob;
  host->set.r2req = p->r2req;
  char *a = (char *)bc->arena + fixed;
  for (int j = 0; j < nprob; j++) {
    BProb &q = host->set.prob[j];
    q.g = gs[j]->l->g;
    q.u = gs[j]->u64;
    q.b = b[j];
    q.x = x[j];
    for (double2 **v : {&q.r, &q.p, &q.ap, &q.t}) {
      *v = (double2 *)a;
      a += vec_bytes(q.g.nh);
    }
    q.m2 = mass[j] * mass[j];
  }
  // the batch runs on its own stream, ordered after the caller's work
  QS_CUDA(cudaStreamSynchronize(stream()));
  const int maxits = p->maxits > 0 ? p->maxits : 50000;
  int per_sm = 1;
  if ((rc = tune(bc, nl, nsets, &per_sm))) return rc;
  *tuned_block = kBatchBlock;
  *tuned_per_sm = per_sm;
  if ((rc = run_batched(bc, nl, per_sm, maxits, true, graph_used))) return rc;
  const std::vector<BState> hs(host->st, host->st + nprob);
  int status = QEXSTAG_OK;
  // FP64 true residuals, all queued before the host waits for the norms (as
  // many at a time as red_results holds); then any problem above its target
  // is defect-corrected (solveXX, stagSolve.nim:330-421)
  std::vector<double> r2s(nprob, 0.0);
  auto views = [&](int j, VecD *rho, VecD *t, VecD *y) -> int {
    qexstag_links_s *g = gs[j];
    const int nh = g->l->g.nh;
    const size_t vb = sizeof(double2) * 3 * (size_t)nh;
    void *prho, *pt, *py;
    int rc2;
    if ((rc2 = g->ws.get(kSlotDcRho, vb, &prho)) || (rc2 = g->ws.get(kSlotTmpOdd, vb, &pt)) ||
        (rc2 = g->ws.get(kSlotDcY, vb, &py)))
      return rc2;
    *rho = VecD{(double2 *)prho, nh};
    *t = VecD{(double2 *)pt, nh};
    *y = VecD{(double2 *)py, nh};
    return QEXSTAG_OK;
  };
  auto residual = [&](int j, const VecD &rho, const VecD &t, double *dev, double *r2) -> int {
    const Geom &geo = gs[j]->l->g;
    int rc2;
    if ((rc2 = schur64(gs[j], 0, rho, CVecD{x[j], geo.V}, t, mass[j] * mass[j])) ||
        (rc2 = vsub(rho, CVecD{b[j], geo.V}, cv(rho), geo.nh)))
      return rc2;
    return dev ? vnorm2_dev(cv(rho), geo.nh, dev) : vnorm2(cv(rho), geo.nh, r2);
  };
  for (int j0 = 0; j0 < nprob; j0 += kNumResults) {
    const int n = std::min(kNumResults, nprob - j0);
    for (int j = j0; j < j0 + n; j++) {
      VecD rho, t, y;
      if ((rc = views(j, &rho, &t, &y)) || (rc = residual(j, rho, t, red_results() + (j - j0), nullptr))) return rc;
    }
    QS_CUDA(cudaMemcpyAsync(host_results(), red_results(), sizeof(double) * n, cudaMemcpyDeviceToHost, stream()));
    QS_CUDA(cudaStreamSynchronize(stream()));
    std::copy(host_results(), host_results() + n, r2s.begin() + j0);
  }
  for (int j = 0; j < nprob; j++) {
    int its = hs[j].itn;
    if (hs[j].b2 == 0.0) {
      iters[j] = 0;
      if (r2_out) r2_out[j] = 0.0;
      continue;
    }
    if (std::isnan(hs[j].r2)) return fail(QEXSTAG_ERR_NAN, "batched solve: NaN residual");
    qexstag_links_s *g = gs[j];
    const Geom &geo = g->l->g;
    const int nh = geo.nh;
    double r2 = r2s[j];
    for (int pass = 0; r2 > p->r2req * hs[j].b2 && its < maxits && pass < 4; pass++) {
      VecD rho, t, y;
      if ((rc = views(j, &rho, &t, &y))) return rc;
      CgOut o{};
      if ((rc = cg64(g, 0, mass[j] * mass[j], cv(rho), y, p->r2req * hs[j].b2 / r2, maxits - its, &o)))
        return rc;
      its += o.iterations;
      st->outer_iterations += 1;
      if ((rc = vaxpy(VecD{x[j], geo.V}, 1.0, cv(y), nh)) || (rc = residual(j, rho, t, nullptr, &r2))) return rc;
    }
    iters[j] = its;
    st->iterations += its;
    const double rel = r2 / hs[j].b2;
    if (r2_out) r2_out[j] = rel;
    st->r2 = std::max(st->r2, rel);
    if (r2 > p->r2req * hs[j].b2) status = QEXSTAG_NOT_CONVERGED;
  }
  return status;
}

}  // namespace qs

using namespace qs;

extern "C" {

int qexstag_barrier_selftest(int missing, double timeout_ms) {
  if (missing < 0 || missing > 1024 || !(timeout_ms > 0.0) || timeout_ms > 10000.0)
    return fail(QEXSTAG_ERR_ARG, "barrier_selftest: missing in [0, 1024], timeout in (0, 10000] ms");
  int rc = runtime_ready();
  if (rc) return rc;
  int dev = 0, khz = 0;
  QS_CUDA(cudaGetDevice(&dev));
  QS_CUDA(cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, dev));
  const long long cycles = (long long)(timeout_ms * (double)khz);  // kHz x ms = cycles
  BGlobal *gl = nullptr;
  int *out = nullptr;
  if (device_malloc(&gl, sizeof(BGlobal)) != cudaSuccess || device_malloc(&out, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    if (gl) cudaFree(gl);
    return fail(QEXSTAG_ERR_ALLOC, "barrier_selftest: allocation failed");
  }
  QS_CUDA(cudaMemsetAsync(gl, 0, sizeof(BGlobal), stream()));
  QS_CUDA(cudaMemsetAsync(out, 0, sizeof(int), stream()));
  // one block per SM: always co-resident, as the cooperative launch checks
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(num_sms());
  cfg.blockDim = dim3(128);
  cfg.stream = stream();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, barrier_selftest_kernel, gl, cycles, (unsigned)missing, out);
  note_launch();
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream());
  int hout = 0, herr = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&hout, out, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&herr, &gl->err, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(gl);
  cudaFree(out);
  if (e != cudaSuccess) return cuda_fail(e, "barrier_selftest");
  if (herr || hout != 1) return fail(QEXSTAG_ERR_TIMEOUT, "barrier_selftest: the grid barrier timed out");
  return QEXSTAG_OK;
}

}  // extern "C"
