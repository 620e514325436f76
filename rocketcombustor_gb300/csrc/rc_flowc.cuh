// How the warps of a dataflow block wait for one another on words of shared
// memory, and the starting warp of the compact launches (k_lusgs_flowc,
// k_lusgs_flowc32).
//
// Several warps write these words while another one polls them, and lanes that
// read for themselves can see different values; what follows from a word holds
// warp-wide votes and barriers.  So every decision is lane 0's (`see`): the
// lanes of a warp take one path by construction.
//
// L is one lane and its primitives (FlowLane in rc_dev.cuh; the tests run the
// same code on processor threads):
//   int lane                         its number
//   static constexpr bool cold       give_up is a call.  The mixed launches run the
//                                    Newton update's code beside the passes' and
//                                    want the waits short (120,000 cells, ten
//                                    iterations 9.67 -> 9.55 ms), the FP64 ones do
//                                    not (20,000 cells 5.38, as a call 5.40)
//   int load(const volatile int*), void store(volatile int*, int)
//   int lane0(int x)                 lane 0's x; void sync(): the warp meets
//   void fence()                     orders shared memory for the block
//   void arrive(int id, int n), void meet(int id, int n)   named barriers
//   void latch()                     records that a wait gave up
//   void nap()                       256 ns at least
//
// Waits are bounded, `limit` units of 256 ns (530 cycles at 2.07 GHz) each or a
// little more, whatever is polled; some warps wait through a whole sweep.  The
// units are counted in polls: 16 of a word in shared memory (59 cycles each), two
// of a flag in memory (280 to 340), one with a nap in between (1,060).  (Read from
// the clock instead, they cost 4 to 8 % of a mixed iteration on 120,000 cells.)
#pragma once

#ifdef __CUDACC__
#define RCF_HD __device__ __forceinline__
#define RCF_COLD __device__ __noinline__
#else
#define RCF_HD inline
#define RCF_COLD inline
#endif

namespace rc {

// polls of a word in shared memory, and of a flag in memory, in a unit of a limit
constexpr unsigned WORD_POLLS = 16, FLAG_POLLS = 2;
// n polls for each of `limit` units, at most 2^32 - 1 in all (two minutes)
RCF_HD unsigned polls_of(unsigned limit, unsigned n) { return limit < 0xffffffffu / n ? n * limit : 0xffffffffu; }

template <class L>
struct WarpWait {
  L l;
  volatile int* bad;  // a wait of the block gave up
  unsigned limit;     // units
  // lane 0's x
  RCF_HD int see(int x) { return l.lane0(x); }
  RCF_HD void give_up() {
    if (L::cold) give_up_cold();
    else give_up_here();
  }
  RCF_COLD void give_up_cold() { give_up_here(); }
  RCF_HD void give_up_here() {
    if (l.lane == 0) {
      l.store(bad, 1);
      l.latch();
    }
    l.sync();
  }
  // Waits until *p >= v; false after a give-up of this wait or of any other.
  RCF_HD bool until(const volatile int* p, int v, bool spaced = false) {
    const unsigned most = polls_of(limit, spaced ? 1u : WORD_POLLS);
    for (unsigned spin = 0;; ++spin) {
      const int s = see((l.load(p) >= v ? 1 : 0) | (l.load(bad) ? 2 : 0));
      if (s) {
        l.fence();
        return s == 1;
      }
      if (spin >= most) {
        give_up();
        return false;
      }
      if (spaced) l.nap();
    }
  }
};

// The compact launches' words: done: passes 0 .. *done - 1 are done;
// ready[k % nbuf] = k + 1: pass k is prepared; go[k & 1]: pass k runs.
template <class L>
struct FlowWarp : WarpWait<L> {
  volatile int *done, *ready, *go;
  int nbuf;
  RCF_HD bool passes_done(int k) { return this->until(done, k + 1); }  // 0 .. k
  RCF_HD void set_ready(int k) {
    this->l.sync();
    this->l.fence();
    if (this->l.lane == 0) this->l.store(ready + k % nbuf, k + 1);
    this->l.sync();
  }
  // The starting warp of a block of n passes.  Barriers 3 and 13 (by the pass's
  // parity) start a pass, 4 and 14 end it, each met by `threads` threads: the
  // compute warps and this one.  A prepared pass is started before the end of
  // the one before has been seen; every pass is started and its end seen,
  // also after a give-up (go = 0 then), so that the barriers stay matched.
  RCF_HD void start_passes(int n, int threads) {
    for (int k = 0; k < n; ++k) {
      const bool early = this->see(this->l.load(ready + k % nbuf) == k + 1);
      if (early) start(k, threads);
      if (k > 0) end(k - 1, threads);
      if (!early) {
        this->until(ready + k % nbuf, k + 1);
        start(k, threads);
      }
    }
    if (n > 0) end(n - 1, threads);
  }

 private:
  RCF_HD void start(int k, int threads) {
    if (this->l.lane == 0) this->l.store(go + (k & 1), this->l.load(this->bad) ? 0 : 1);
    this->l.sync();
    this->l.fence();
    this->l.arrive(3 + 10 * (k & 1), threads);
  }
  RCF_HD void end(int k, int threads) {
    this->l.meet(4 + 10 * (k & 1), threads);
    this->l.fence();
    if (this->l.lane == 0) this->l.store(done, k + 1);
    this->l.sync();
  }
};

}  // namespace rc
