// The staged stream of the tiled wavelets (csrc/stages.cuh) run by host threads,
// one a lane, with mbarriers and barriers of their own: a wait that runs
// out, in thread 0's refill or in one lane, must leave no lane waiting for another
// for good, and every copy issued must have landed at the end; no copy may be
// issued into a stage that a lane has read without a proxy fence, after the lane's
// warp released the stage, since.  Exits nonzero on a failure.
#include "stages.cuh"

#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

using namespace std::chrono_literals;

namespace {

constexpr int kWarps = 2, kLanes = 32 * kWarps;
constexpr auto kWait = 600ms;     // a bounded wait on an mbarrier
constexpr auto kHang = 5000ms;    // lanes that meet later than this never do

struct Left {};  // a lane gave up on a barrier that nobody will complete

std::mutex mu;
std::condition_variable cv;

struct Bar { int count = 0, pending = 0, phase = 0; };
std::map<uint64_t*, Bar> bars;
void arrive_locked(Bar& b) {
  if (--b.pending == 0) {
    b.pending = b.count;
    ++b.phase;
    cv.notify_all();
  }
}

struct Meet {  // a barrier of n threads
  int n = 0, here = 0, gen = 0;
  void operator()() {
    std::unique_lock<std::mutex> lk(mu);
    const int g = gen;
    if (++here == n) {
      here = 0;
      ++gen;
      cv.notify_all();
      return;
    }
    if (!cv.wait_for(lk, kHang, [&] { return gen != g; })) throw Left{};
  }
};
Meet warp_meet[kWarps], cta_meet;

thread_local int tid;
// the stages a lane has read with no fence since, and those its warp has released
unsigned unfenced[kLanes], released[kWarps];
std::map<uint64_t*, int> stage_of_empty;
std::function<bool(uint64_t*, unsigned)> runs_out;  // the wait of this thread that is made to fail

struct Sim {
  static void init(uint64_t* bar, unsigned count) { bars[bar] = Bar{(int)count, (int)count, 0}; }
  static void init_done() {}
  static bool wait(uint64_t* bar, unsigned phase) {
    std::unique_lock<std::mutex> lk(mu);
    if (runs_out(bar, phase)) return false;
    return cv.wait_for(lk, kWait, [&] { return (unsigned)(bars[bar].phase & 1) != phase; });
  }
  static void arrive(uint64_t* bar) {
    std::lock_guard<std::mutex> g(mu);
    released[tid / 32] |= 1u << stage_of_empty.at(bar);
    arrive_locked(bars[bar]);
  }
  static void refill_fence() {
    std::lock_guard<std::mutex> g(mu);
    for (int l = 0; l < kLanes; ++l) unfenced[l] &= ~released[l / 32];
  }
  static void sync() { warp_meet[tid / 32](); }
};

// the copy engine: chunks land a little after they were issued
struct Copy { uint64_t* bar; int* dst; int value; };
std::deque<Copy> copies;
bool stop = false;
void engine() {
  std::unique_lock<std::mutex> lk(mu);
  while (!stop || !copies.empty()) {
    if (copies.empty()) {
      cv.wait_for(lk, 1ms);
      continue;
    }
    const Copy c = copies.front();
    lk.unlock();
    std::this_thread::sleep_for(300us);
    lk.lock();
    copies.pop_front();
    *c.dst = c.value;
    arrive_locked(bars[c.bar]);
  }
}

// which: 0 no wait fails, 1 thread 0's refill wait, 2 one lane's wait for its data
template <int STAGES, int LAG>
int run(int nch, int which) {
  uint64_t bar[2 * STAGES];
  int stage[STAGES], fail = 0, err = 0, hung = 0, wrong = 0, in_flight = 0, unordered = 0;
  for (unsigned& u : unfenced) u = 0;
  for (unsigned& u : released) u = 0;
  for (int q = 0; q < STAGES; ++q) stage_of_empty[&bar[STAGES + q]] = q;
  for (int& v : stage) v = -1;
  bars.clear();
  for (Meet& m : warp_meet) m = Meet{32};
  cta_meet = Meet{kLanes};
  copies.clear();
  stop = false;
  bool fired = false;
  runs_out = [&](uint64_t* b, unsigned) {
    const bool refill = b >= bar + STAGES;
    if (fired || fail) return false;
    if ((which == 1 && refill && tid == 0) || (which == 2 && !refill && tid == 37 && b == bar + 1)) return fired = true;
    return false;
  };
  std::thread eng(engine);
  std::vector<std::thread> lanes;
  for (int t = 0; t < kLanes; ++t)
    lanes.emplace_back([&, t] {
      tid = t;
      try {
        stl::StageStream<Sim, STAGES, LAG, kWarps> cs(bar, bar + STAGES);
        cs.nch = nch;
        auto issue = [&](int c) {
          std::lock_guard<std::mutex> g(mu);
          for (unsigned u : unfenced) unordered += u >> (c % STAGES) & 1;
          copies.push_back({&bar[c % STAGES], &stage[c % STAGES], c});
          cv.notify_all();
        };
        if (tid == 0) {
          cs.init();
          cs.begin(nch, issue);
        }
        cta_meet();
        for (int c = 0; c < nch; ++c) {
          if (cs.wait(c)) {
            std::lock_guard<std::mutex> g(mu);
            wrong += stage[c % STAGES] != c;
            unfenced[tid] |= 1u << (c % STAGES);
            released[tid / 32] &= ~(1u << (c % STAGES));
          }
          Sim::sync();  // the slots of the adjoint
          cs.release(c, tid, issue);
        }
        if (!cs.ok) {
          std::lock_guard<std::mutex> g(mu);
          fail = 1;
        }
        cta_meet();
        if (fail && tid == 0) err = cs.drain();
        if (tid == 0) {
          std::lock_guard<std::mutex> g(mu);
          in_flight = (int)copies.size();
        }
      } catch (Left) {
        std::lock_guard<std::mutex> g(mu);
        ++hung;
      }
    });
  for (auto& l : lanes) l.join();
  {
    std::lock_guard<std::mutex> g(mu);
    stop = true;
  }
  eng.join();
  const int want = which && nch > STAGES + LAG ? stl::kErrWait : 0;
  const bool good = !hung && !wrong && !in_flight && !unordered && err == want && (want ? fired : !fail);
  if (!good)
    std::printf("stages %d lag %d chunks %d case %d: %d lanes left waiting, %d wrong reads, %d copies in flight, "
                "%d reads not ordered before a copy, error %d (%d)\n",
                STAGES, LAG, nch, which, hung, wrong, in_flight, unordered, err, want);
  return !good;
}

}  // namespace

int main() {
  int fails = 0;
  for (int which : {0, 1, 2}) {
    fails += run<3, 1>(9, which);  // the grid wavelets
    fails += run<2, 0>(7, which);  // the coloured forward
  }
  for (int nch : {0, 1, 2, 3, 4}) fails += run<3, 1>(nch, 0) + run<2, 0>(nch, 0);
  std::printf("fails %d\n", fails);
  return fails != 0;
}
