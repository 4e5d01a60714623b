// The rounds of a neighbour search over one window column (a range of the sorted particles): each
// round takes CAND_STEP consecutive candidates. A warp's lanes go through their particles' columns
// together, for as many rounds as the longest of them needs, and every lane loads its candidate
// records in every one of them without a test, so that the loads of a round are independent. (Plain
// C++, so that the index arithmetic also runs on the host.)
#pragma once

#ifdef __CUDACC__
#define MF_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MF_HOST_DEVICE inline
#endif

namespace mf {

constexpr int CAND_STEP = 8;  // candidates per particle and round
// Records the arrays of candidate records are longer than their N particles: a round starts at
// N at the latest and loads CAND_STEP records, of which those past the column's end are not used.
constexpr int CAND_PAD = CAND_STEP;

// The start of the round after the one at jb. A lane whose column has ended starts further on, and
// at N in the end, while its warp's other lanes finish theirs: without the limit it ran past the
// records by as many rounds as the longest column had more than its own.
MF_HOST_DEVICE int next_round(int jb, int N) {
  const int next = jb + CAND_STEP;
  return next < N ? next : N;
}

}  // namespace mf
