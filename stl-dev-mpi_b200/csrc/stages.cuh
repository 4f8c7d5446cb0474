// The staged coefficient stream of the tiled wavelets: the chunks of a CTA pass
// through STAGES stages of shared memory, chunk c through stage c % STAGES.
// Thread 0 fills the stages by bulk asynchronous copies; every warp waits for a
// stage on its own, reads it and releases it with one arrival; thread 0 refills
// the stage of chunk c - LAG after it released chunk c (LAG 1: the other warps have had a
// chunk's time to release it, so the refill seldom waits).
//
// Every wait is bounded, and no lane leaves the chunks early: a wait that ran out
// (thread 0's for a free stage among them) clears the thread's ok, it waits and
// issues no more, and goes through the remaining chunks' barriers with its
// warp.  Lanes that left alone would wait at the CTA's barrier while the rest of
// their warp waits for them at the next __syncwarp.  The results of such a CTA are
// not used.  A thread that is not ok may see a stage in any state.
//
// The stages are read by ordinary loads and written by the copy engine, another
// proxy: a barrier orders the two only together with a proxy fence on the way from
// the reads to the copy.  Thread 0 executes it between its wait for the readers'
// releases and the refill.  (One by every reader before its release orders the same
// accesses and measured slower: 2.76 -> 2.82 ms for the FP64 adjoints at nside 512, J 8.)
//
// P supplies the mbarriers, the fence and the warp's barrier: the device's in
// kernels.cu, threads that check for lanes left behind in the host test.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define STL_STAGE_FN __device__ __forceinline__
#else
#define STL_STAGE_FN inline
#endif

namespace stl {

// error flag of a launch: a wait ran out and the copies in flight then landed, or
// they did not
constexpr int kErrWait = 1, kErrDrain = 2;

template <class P, int STAGES, int LAG, int WARPS>
struct StageStream {
  uint64_t *full, *empty;  // [STAGES]: a stage's copies have landed; every warp has read it
  int nch = 0;             // chunks
  int issued = 0;          // chunks issued (thread 0)
  bool ok = true;          // no wait of this thread ran out
  STL_STAGE_FN StageStream(uint64_t* f, uint64_t* e) : full(f), empty(e) {}
  STL_STAGE_FN void init() {  // thread 0, before the first issue and the CTA's barrier
    for (int q = 0; q < STAGES; ++q) {
      P::init(&full[q], 1);
      P::init(&empty[q], WARPS);
    }
    P::init_done();
  }
  // thread 0: issue(c) queues the copies of chunk c into its stage
  template <class F>
  STL_STAGE_FN void begin(int chunks, F&& issue) {
    for (; issued < chunks && issued < STAGES; ++issued) issue(issued);
  }
  // whether chunk c has landed
  STL_STAGE_FN bool wait(int c) { return ok = ok && P::wait(&full[c % STAGES], (unsigned)(c / STAGES) & 1); }
  // after the warp read chunk c
  template <class F>
  STL_STAGE_FN void release(int c, int tid, F&& issue) {
    P::sync();
    if ((tid & 31) == 0) P::arrive(&empty[c % STAGES]);
    const int d = c - LAG;
    if (tid == 0 && ok && d >= 0 && d + STAGES < nch) {
      ok = P::wait(&empty[d % STAGES], (unsigned)(d / STAGES) & 1);
      if (ok) {
        P::refill_fence();
        issue(d + STAGES);
        issued = d + STAGES + 1;
      }
    }
  }
  // thread 0, after a wait ran out anywhere: the copies in flight land (bounded)
  STL_STAGE_FN int drain() {
    bool landed = true;
    for (int q = issued > STAGES ? issued - STAGES : 0; q < issued; ++q)
      landed &= P::wait(&full[q % STAGES], (unsigned)(q / STAGES) & 1);
    return landed ? kErrWait : kErrDrain;
  }
};

}  // namespace stl
