// batch_part.cuh -- how the batched solver's blocks share its problems (also
// compiled for the host alone, by the test of its bounds).
#pragma once

#ifdef __CUDACC__
#define QS_HOST_DEVICE __host__ __device__
#else
#define QS_HOST_DEVICE
#endif

namespace qs {

constexpr int kMaxBatch = 128;  // problems of a batch

// Problems that one block's chunk can meet, for which a block has room: all of
// them.  Chunks are equal in sets of sites, so a few large lattices make a chunk
// that takes in every small one (127 of 4^4 beside one of 48^4).
constexpr int kMaxMet = kMaxBatch;

// The partition: the still-active problems (ids, in order), soff[i] the first
// set of the i-th, cut into equal contiguous chunks, one to each of the first
// nb blocks.  Every block builds the same table.
struct BPart {
  int na;      // active problems
  int ntot;    // their sets
  int nb;      // blocks with a chunk
  int s0, s1;  // this block's sets
  int i0, np;  // the first problem that it meets, and how many
  int ids[kMaxBatch];
  int soff[kMaxBatch + 1];
};

// block b's table of nprob problems, of which those with done(j) are left out
// and j has sets(j) sets; blocks in all
template <class Done, class Sets>
QS_HOST_DEVICE inline void fill_part(BPart &T, int nprob, Done done, Sets sets, int blocks, int b) {
  int n = 0, off = 0;
  for (int j = 0; j < nprob; j++) {
    if (done(j)) continue;
    T.ids[n] = j;
    T.soff[n] = off;
    off += sets(j);
    n++;
  }
  T.soff[n] = off;
  T.na = n;
  T.ntot = off;
  T.nb = blocks < off ? blocks : off;
  T.s0 = b < T.nb ? (int)((long long)b * off / T.nb) : off;
  T.s1 = b < T.nb ? (int)((long long)(b + 1) * off / T.nb) : off;
  T.i0 = T.np = 0;
  if (T.s0 < T.s1) {
    while (T.soff[T.i0 + 1] <= T.s0) T.i0++;
    T.np = 1;
    while (T.soff[T.i0 + T.np] < T.s1) T.np++;
  }
}

// the block whose chunk holds set s
QS_HOST_DEVICE inline int block_of(const BPart &T, int s) {
  return (int)(((long long)(s + 1) * T.nb - 1) / T.ntot);
}

}  // namespace qs
