// The waits of a dataflow block's warps (csrc/rc_flowc.cuh) on processor
// threads: 32 threads are the lanes of a warp.  Every warp-wide operation is a
// meeting of the lanes at one place of the code; lanes that meet at different
// places are counted as a mismatch (on the GPU: a hang or worse).
//
// The words change between the lanes' reads: whenever lanes 1-31 read a word,
// they first wait until it has moved on from what lane 0 read, as long as
// another thread is about to move it.  With PER_LANE (the mistake that the
// check has to notice) each lane decides by its own reading.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "rc_flowc.cuh"

using Clock = std::chrono::steady_clock;
struct Mismatch {};
// how long lanes wait for one another: with PER_LANE some never come
#ifdef PER_LANE
constexpr std::chrono::seconds PATIENCE(3);
#else
constexpr std::chrono::seconds PATIENCE(60);
#endif
static std::atomic<bool> failed{false};
static long mismatches = 0, errors = 0;

// until f(), at most PATIENCE; false then
static bool soon(const std::function<bool()>& f) {
  const auto end = Clock::now() + PATIENCE;
  while (!f()) {
    if (failed || Clock::now() > end) return false;
    std::this_thread::yield();
  }
  return true;
}

// The lanes' meeting place: all 32 bring the same tag, and get lane 0's value.
struct Meeting {
  std::mutex mu;
  std::condition_variable cv;
  int count = 0, tag = 0, value[2] = {};
  unsigned round = 0;
  int come(int lane, int t, int v) {
    std::unique_lock<std::mutex> lock(mu);
    if (failed) throw Mismatch();
    const unsigned r = round;
    if (count == 0) tag = t;
    if (lane == 0) value[r & 1] = v;
    if (tag != t) failed = true;
    if (++count == 32) {
      count = 0;
      ++round;
    }
    if (failed || round != r) cv.notify_all();
    if (!cv.wait_for(lock, PATIENCE, [&] { return failed || round != r; })) {
      failed = true;
      cv.notify_all();
    }
    if (failed) throw Mismatch();
    return value[r & 1];
  }
};

struct Block {
  static constexpr int NBUF = 6;
  std::atomic<int> bad{0}, done{0}, ready[NBUF], go[2], latched{0};
  std::atomic<long> looked{0};  // lane 0's readings
  std::atomic<int> started[2], ended[2];
  Meeting m;
  Block() {
    for (auto& r : ready) r = 0;
    for (int p = 0; p < 2; ++p) { go[p] = 0; started[p] = 0; ended[p] = 0; }
  }
};
static Block* B;
static std::atomic<bool> moving{false};  // the words are about to move

struct Lane {
  static constexpr bool cold = false;
  int lane;
  static std::atomic<int>* word(const volatile int* p) {
    return reinterpret_cast<std::atomic<int>*>(const_cast<int*>(p));
  }
  int load(const volatile int* p) const {
    if (lane == 0) {
      const int x = *word(p);
      seen = x;
      ++B->looked;
      return x;
    }
    for (int k = 0; k < 200 && moving && *word(p) == seen; ++k) std::this_thread::yield();
    return *word(p);
  }
  void store(volatile int* p, int v) const { *word(p) = v; }
  mutable long polls = 0;
#ifdef PER_LANE
  int lane0(int x) const { return x; }
#else
  int lane0(int x) const {
    ++polls;
    return B->m.come(lane, 1, x);
  }
#endif
  void sync() const { B->m.come(lane, 2, 0); }
  void fence() const {}
  void arrive(int id, int) const {
    B->m.come(lane, 100 + id, 0);
    if (lane == 0 && ++B->started[id / 10] != 1) ++errors;
    B->m.come(lane, 200 + id, 0);
  }
  void meet(int id, int) const {
    B->m.come(lane, 300 + id, 0);
    if (lane == 0) {
      if (!soon([&] { return B->ended[id / 10] == 1; })) ++errors;
      B->ended[id / 10] = 0;
    }
    B->m.come(lane, 400 + id, 0);
  }
  void latch() const { ++B->latched; }
  void nap() const { std::this_thread::yield(); }
  static std::atomic<int> seen;
};
std::atomic<int> Lane::seen{0};

static volatile int* raw(std::atomic<int>& a) { return reinterpret_cast<volatile int*>(&a); }
static rc::FlowWarp<Lane> warp_of(int lane, unsigned limit) {
  return {{Lane{lane}, raw(B->bad), limit}, raw(B->done), raw(B->ready[0]), raw(B->go[0]), Block::NBUF};
}
static void lanes(const std::function<void(int)>& f) {
  std::vector<std::thread> t;
  std::atomic<int> caught{0};
  for (int l = 0; l < 32; ++l)
    t.emplace_back([&, l] {
      try {
        f(l);
      } catch (Mismatch&) {
        ++caught;
      }
    });
  for (auto& x : t) x.join();
  if (caught) ++mismatches;
}

// A block of n passes: the starting warp's lanes, one thread that prepares the
// passes at the worst moments, one that runs them.
static void starting_warp(int n) {
  Block b;
  B = &b;
  failed = false;
  int ran = 0;
  std::thread prepare([&] {
    for (int k = 0; k < n; ++k) {
      if (!soon([&] { return b.done >= k - Block::NBUF + 1; })) return;
      moving = true;
      if (k % 3) {  // between lane 0's reading and the others'
        const long at = b.looked;
        soon([&] { return b.looked > at || b.done >= n; });
      }
      b.ready[k % Block::NBUF] = k + 1;
    }
    moving = false;
  });
  std::thread compute([&] {
    for (int k = 0; k < n; ++k) {
      if (!soon([&] { return b.started[k & 1] == 1; })) return;
      b.started[k & 1] = 0;
      if (!b.go[k & 1] || b.ready[k % Block::NBUF] != k + 1) ++errors;
      ++ran;
      b.ended[k & 1] = 1;
    }
  });
  lanes([&](int l) { warp_of(l, 1u << 30).start_passes(n, 64); });
  prepare.join();
  compute.join();
  if (!failed && (ran != n || b.done != n)) ++errors;
}

// A wait that ends as another warp's gives up, at the worst moment.
static void give_up_beside(int n) {
  for (int k = 0; k < n; ++k) {
    Block b;
    B = &b;
    failed = false;
    moving = true;
    std::thread other([&] {
      const long at = b.looked;
      soon([&] { return b.looked > at + k; });
      if (k & 1) b.done = 1;
      b.bad = 1;
      moving = false;
    });
    std::atomic<int> yes{0};
    lanes([&](int l) {
      auto w = warp_of(l, 1u << 30);
      if (w.passes_done(0)) ++yes;
      else w.l.sync();
    });
    other.join();
    if (!failed && yes != 0 && yes != 32) ++errors;
  }
}

// A wait that runs out: false in every lane, one report, and not before its
// `limit` units of 256 ns (530 cycles) for polls of a load and a shuffle, 40
// cycles at least.
static void runs_out() {
  Block b;
  B = &b;
  failed = false;
  moving = false;
  std::atomic<int> yes{0}, early{0};
  lanes([&](int l) {
    auto w = warp_of(l, 50);
    if (w.passes_done(0)) ++yes;
    if (w.l.polls * 40 < 50 * 530) ++early;
  });
  if (!failed && (yes != 0 || early != 0 || b.latched != 1 || b.bad != 1)) ++errors;
}

int main() {
  starting_warp(60);
  give_up_beside(8);
  runs_out();
  std::printf("mismatches %ld errors %ld\n", mismatches, errors);
  return mismatches || errors;
}
