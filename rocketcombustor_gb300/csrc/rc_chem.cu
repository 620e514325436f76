// Chemistry integrator kernels (FP64, --fmad=false): the integrated chemical
// source of the steady iteration and the batch integration of given states.
//
// The work per cell is uneven (1 to maxsub substeps, each with rejections), so
// the kernels are persistent work queues: every lane takes the next item from
// a counter when it has finished one.  Results do not depend on which lane
// takes which item.
#include <cuda_runtime.h>

#include "rc_chem.cuh"
#include "rc_dev.cuh"

namespace rc {

constexpr int CHEM_THREADS = 128;
using ChemNum = Num<false>;

// Runs the items 0 .. n-1 of a queue through the lanes of a warp: a lane that
// has finished its item takes the next one while the others go on.  Items need
// 1 to thousands of attempts; a warp that took 32 and waited for the slowest
// left most lanes idle (an FP64 instruction costs the same with one active lane
// as with 32).  The lanes refill when REFILL of them are idle or none is busy:
// starting an item costs about a tenth of an attempt, for the whole warp.
// 262,144 states at tolerance 0.005 (median 9 substeps, 90th percentile 509):
// 276 ms with a warp taking 32 states at a time, 113 ms with the queue.
//
// That leaves the end of the queue: every warp then holds a few long items,
// each attempt at the price of a full warp.  So the integration goes in rounds
// (launches): a round gives its items, through full warps, at most park_at(round)
// attempts in all and parks what is left of them in a list in memory, which is the
// next round's queue.  Of unsorted items (park.cut) a round that has more than the
// launch has lanes ends when its queue is empty: the items in the lanes are
// parked as they are, at the end of the list, and since a list is taken from its
// end, they go first in the next round.  The last round ends with its items.
// Where the list is full the items stay in their lanes.  The same states: 74 ms.
// One / two / four / ten rounds, ms: tolerance 0.05, 65,536 states 7.7 / 6.1 / 6.2 /
// 6.2, 262,144 17.2 / 13.8 / 13.7 / 13.7; 0.005, 30,000 34.5 / 27.9 / 27.9 / 28.0,
// 131,072 57.8 / 55.2 / 55.2 / 50.8.  The kernels spill 434-462 bytes at the 168
// registers that three blocks per SM leave a thread.
//   begin(item, r)  loads item into reactor r; false when it needs no attempt
//   end(item, r)    stores the finished item
constexpr int REFILL = 4;
__host__ __device__ constexpr int park_at(int round) { return round == 0 ? 16 : 64 * round; }

// list l of the parked reactors: their items and their state
template <int NSP, class N>
struct Parked {
  static constexpr int V = 3 + NSP;
  double* x;
  int* k;
  size_t cap;
  __device__ __forceinline__ Parked(const ChemPark& p, int l)
      : x(p.x + (size_t)l * CHEM_PARK_X * p.cap), k(p.k + (size_t)l * CHEM_PARK_K * p.cap), cap(p.cap) {}
  __device__ __forceinline__ void put(size_t u, int item, const Reactor<NSP, N>& r) const {
    static_assert(V + 4 <= CHEM_PARK_X, "room for the state");
#pragma unroll
    for (int v = 0; v < V; ++v) x[v * cap + u] = val(r.P[v]);
    x[V * cap + u] = val(r.rho);
    x[(V + 1) * cap + u] = val(r.e);
    x[(V + 2) * cap + u] = val(r.rem);
    x[(V + 3) * cap + u] = val(r.hs);
    k[u] = item;
    k[cap + u] = r.nacc;
    k[2 * cap + u] = r.natt;
  }
  __device__ __forceinline__ int get(size_t u, Reactor<NSP, N>& r) const {
#pragma unroll
    for (int v = 0; v < V; ++v) r.P[v] = x[v * cap + u];
    r.rho = x[V * cap + u];
    r.e = x[(V + 1) * cap + u];
    r.rem = x[(V + 2) * cap + u];
    r.hs = x[(V + 3) * cap + u];
    r.nacc = k[cap + u];
    r.natt = k[2 * cap + u];
    return k[u];
  }
};

// Round 0 takes the items 0 .. n-1, a later round the list of the one before;
// the first 32 of a warp are its own (so that few items spread over the blocks
// in order), the others come from the round's counter.
// LISTED: a round with at most one item per lane is the last.
template <int NSP, class N, bool LISTED, class Begin, class End>
__device__ __forceinline__ void run_queue(const ThermoDev<NSP>& th, int n, const ChemPark& park, int round, double tol,
                                          int maxsub, unsigned& err, Begin begin, End end) {
  const int lane = threadIdx.x & 31;
  const Parked<NSP, N> from(park, (round + 1) & 1), to(park, round & 1);
  if (round > 0) n = (int)min(park.count[CHEM_ROUNDS + round - 1], (unsigned)park.cap);
  const int lanes = gridDim.x * CHEM_THREADS;
  const bool final = round + 1 >= park.rounds || (LISTED && n <= lanes);
  const int limit = final ? 0x7fffffff : park_at(round);
  Reactor<NSP, N> r;
  int item = -1;        // the lane's item, -1 when idle
  bool more = true;     // the queue may hold more (warp-uniform)
  bool first = true, full = false;
  for (;;) {
    unsigned idle = __ballot_sync(0xffffffffu, item < 0);
    while (more && (__popc(idle) >= REFILL)) {
      int base = blockIdx.x * CHEM_THREADS + (threadIdx.x & ~31);
      if (!first) {
        if (lane == 0) base = lanes + (int)atomicAdd(park.count + round, (unsigned)__popc(idle));
        base = __shfl_sync(0xffffffffu, base, 0);
      }
      first = false;
      more = base + __popc(idle) < n;
      if (item < 0) {
        const int q = base + __popc(idle & ((1u << lane) - 1u));
        if (q < n) {
          if (round > 0) {
            item = from.get(n - 1 - q, r);
          } else {
            item = q;
            if (!begin(q, r)) {
              end(q, r);
              item = -1;
            }
          }
        }
      }
      __syncwarp();
      idle = __ballot_sync(0xffffffffu, item < 0);
    }
    if (idle == 0xffffffffu) break;
    // the queue is empty, in a round that had more items than lanes
    const bool stop = park.cut && !final && n > lanes && lanes + (int)*(volatile unsigned*)(park.count + round) >= n;
    if (item >= 0) {
      if (!r.attempt(th, tol, maxsub, err)) {
        end(item, r);
        item = -1;
      } else if (!final && (stop || r.natt >= limit) && !full) {
        const unsigned u = atomicAdd(park.count + CHEM_ROUNDS + round, 1u);
        full = u >= (unsigned)park.cap;
        if (!full) {
          to.put(u, item, r);
          item = -1;
        }
      }
    }
    __syncwarp();
  }
}

// Integrated source of cell i (sourceterm.f90:43-51 with omega replaced by
// the mean rate over the cell's pseudo time step):
//   src_k = vol * (rho * ((Y_k(step) - Y_k) / step)), with the reactor's rho = p / (R_mix T).
template <int NSP, class N, bool LISTED, class Cell>
__device__ __forceinline__ void run_cells(const Dev& d, const ThermoDev<NSP>& th, int n, Cell cell, double tol,
                                          int maxsub, int* nsub, const ChemPark& park, int round) {
  constexpr int V = 3 + NSP;
  const int NE = d.NE;
  unsigned err = 0;
  run_queue<NSP, N, LISTED>(
      th, n, park, round, tol, maxsub, err,
      [&](int q, Reactor<NSP, N>& r) {
        const int i = cell(q);
#pragma unroll
        for (int k = 0; k < V; ++k) r.P[k] = d.PA[k * NE + i];
        return r.begin(th, N(d.step[i]), err);
      },
      [&](int q, const Reactor<NSP, N>& r) {
        const int i = cell(q);
        nsub[i] = r.nacc;
        const N dt = d.step[i];
        const double vol = d.vol[i];
#pragma unroll
        for (int k = 0; k < NSP - 1; ++k)
          d.src[k * NE + i] = val(vol * (r.rho * ((r.P[4 + k] - d.PA[(4 + k) * NE + i]) / dt)));
      });
  flag(d, err);
}

// Cells are taken in `order` (longest previous integration first, so the long
// cells start early), or in cell order when order is null.
template <int NSP, class N>
__global__ void __launch_bounds__(CHEM_THREADS, 3) k_chem_source(const Dev d, const ThermoDev<NSP> th, double tol,
                                                              int maxsub, int* __restrict__ nsub,
                                                              const int* __restrict__ order, const ChemPark park, int round) {
  run_cells<NSP, N, false>(d, th, d.NE, [&](int q) { return order ? order[q] : q; }, tol, maxsub, nsub, park, round);
}

// Counting sort of the cells by their previous substep count, descending
// (bucket 255 - min(nsub, 255)); the order inside a bucket does not matter.
// Most cells share a few counts (1, or the cap), so the counting is aggregated:
// the lanes of a warp that hold one bucket add once, in shared memory, and a
// block adds its non-empty buckets to the global counters (one global atomic
// per cell on the same address took 0.6 ms per kernel on a million cells).
constexpr int NBUCKET = 256, SORT_ITEMS = 8;  // items per thread of the NBUCKET-thread sort blocks
__device__ __forceinline__ int chem_bucket(int n) { return NBUCKET - 1 - min(max(n, 0), NBUCKET - 1); }
// adds the warp's `in` lanes to cnt[bucket]; each lane's place in the bucket
__device__ __forceinline__ unsigned bucket_add(unsigned* cnt, int bucket, bool in) {
  const int lane = threadIdx.x & 31;
  const unsigned act = __ballot_sync(0xffffffffu, in);
  unsigned place = 0;
  if (in) {
    const unsigned m = __match_any_sync(act, bucket);
    unsigned base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(&cnt[bucket], (unsigned)__popc(m));
    place = __shfl_sync(m, base, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
  }
  __syncwarp();
  return place;
}
__global__ void __launch_bounds__(NBUCKET) k_chem_hist(const int* __restrict__ nsub, int n, unsigned* hist) {
  __shared__ unsigned cnt[NBUCKET];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int u = 0; u < SORT_ITEMS; ++u) {
    const int i = (blockIdx.x * SORT_ITEMS + u) * NBUCKET + threadIdx.x;
    bucket_add(cnt, i < n ? chem_bucket(nsub[i]) : 0, i < n);
  }
  __syncthreads();
  if (cnt[threadIdx.x]) atomicAdd(&hist[threadIdx.x], cnt[threadIdx.x]);
}
__global__ void k_chem_scan(unsigned* hist) {  // one block of NBUCKET threads: exclusive scan in place
  __shared__ unsigned sh[NBUCKET];
  const int t = threadIdx.x;
  sh[t] = hist[t];
  __syncthreads();
  for (int o = 1; o < NBUCKET; o <<= 1) {
    const unsigned v = t >= o ? sh[t - o] : 0u;
    __syncthreads();
    sh[t] += v;
    __syncthreads();
  }
  hist[t] = t ? sh[t - 1] : 0u;
}
__global__ void __launch_bounds__(NBUCKET) k_chem_scatter(const int* __restrict__ nsub, int n, unsigned* cursor,
                                                          int* __restrict__ order) {
  __shared__ unsigned cnt[NBUCKET], base[NBUCKET];
  cnt[threadIdx.x] = 0;
  __syncthreads();
  unsigned place[SORT_ITEMS];
  int bucket[SORT_ITEMS];
#pragma unroll
  for (int u = 0; u < SORT_ITEMS; ++u) {
    const int i = (blockIdx.x * SORT_ITEMS + u) * NBUCKET + threadIdx.x;
    bucket[u] = i < n ? chem_bucket(nsub[i]) : 0;
    place[u] = bucket_add(cnt, bucket[u], i < n);
  }
  __syncthreads();
  base[threadIdx.x] = cnt[threadIdx.x] ? atomicAdd(&cursor[threadIdx.x], cnt[threadIdx.x]) : 0u;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < SORT_ITEMS; ++u) {
    const int i = (blockIdx.x * SORT_ITEMS + u) * NBUCKET + threadIdx.x;
    if (i < n) order[base[bucket[u]] + place[u]] = i;
  }
}

// The same for the cells list[0 .. *nlist) (the surrogate's fallbacks).
template <int NSP, class N>
__global__ void __launch_bounds__(CHEM_THREADS, 3) k_chem_list(const Dev d, const ThermoDev<NSP> th, double tol,
                                                            int maxsub, int* __restrict__ nsub,
                                                            const int* __restrict__ list,
                                                            const unsigned* __restrict__ nlist, const ChemPark park,
                                                            int round) {
  run_cells<NSP, N, true>(d, th, (int)min(*nlist, (unsigned)d.NE), [&](int q) { return list[q]; }, tol, maxsub, nsub,
                    park, round);
}

// n primitive states in SoA ([k*n + i]) integrated over dt[i].
template <int NSP, class N>
__global__ void __launch_bounds__(CHEM_THREADS, 3) k_chem_batch(const ThermoDev<NSP> th, const double* __restrict__ Pin,
                                                             const double* __restrict__ dts, int n,
                                                             double* __restrict__ Pout, int* __restrict__ nsub,
                                                             double tol, int maxsub, const ChemPark park,
                                                             int round, unsigned* errp) {
  constexpr int V = 3 + NSP;
  unsigned err = 0;
  run_queue<NSP, N, false>(
      th, n, park, round, tol, maxsub, err,
      [&](int i, Reactor<NSP, N>& r) {
#pragma unroll
        for (int k = 0; k < V; ++k) r.P[k] = Pin[(size_t)k * n + i];
        return r.begin(th, N(dts[i]), err);
      },
      [&](int i, const Reactor<NSP, N>& r) {
        nsub[i] = r.nacc;
#pragma unroll
        for (int k = 0; k < V; ++k) Pout[(size_t)k * n + i] = val(r.P[k]);
      });
  if (err) atomicOr(errp, err);
}

// Grid of the persistent launches: enough resident warps to fill every SM.
template <class K>
static int chem_grid(K kernel, int items, int* nsm) {
  int dev = 0, occ = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, CHEM_THREADS, 0);
  const int need = (items + CHEM_THREADS - 1) / CHEM_THREADS;
  const int g = (*nsm > 0 ? *nsm : 1) * (occ > 0 ? occ : 1);
  return g < need ? g : (need > 0 ? need : 1);
}
// The rounds of a launch over `items`: one where there is no room to park, or
// where one block per SM holds all items (a warp without neighbours on its
// sub-partition has nothing to gain from full lanes).  Items that come sorted,
// the longest of the last iteration first, need few: the last ones to start are
// short (64 cases, a million cells, five iterations: 139.3 ms in one round, 137.5
// in four, 140.7 in ten with the cut; unsorted states: 113, 101 and 74 ms).  How
// many items a list on the device holds is known there only, and often there are
// none: it goes in three rounds, and a round that has no more items than the
// launch has lanes ends with them (an iteration with the surrogate and all cells
// in the list, one / two / three / ten rounds, ms: 30,000 cells 11.30 / 11.52 / 11.32 /
// 11.75; 120,000 15.19 / 15.42 / 15.22 / 15.57; 600,000 51.98 / 50.07 / 49.20 / 49.25).
enum ChemItems { CHEM_UNSORTED, CHEM_SORTED, CHEM_LISTED };
template <class K, class Launch>
static int chem_rounds(K kernel, int items, ChemItems kind, ChemPark park, cudaStream_t s, Launch launch) {
  int nsm = 0;
  const int grid = chem_grid(kernel, items, &nsm);
  park.rounds = kind == CHEM_SORTED ? 4 : kind == CHEM_LISTED ? 3 : CHEM_ROUNDS;
  if (park.cap == 0 || items <= nsm * CHEM_THREADS) park.rounds = 1;
  park.cut = kind != CHEM_SORTED;
  cudaMemsetAsync(park.count, 0, sizeof(unsigned) * 2 * CHEM_ROUNDS, s);
  for (int round = 0; round < park.rounds; ++round) launch(grid, park, round);
  return park.rounds;
}

// order/hist: work arrays of NE ints and NBUCKET unsigned (order null: cell order)
template <int NSP>
int chem_source(const Dev& d, const void* th, double tol, int maxsub, int* nsub, int* order, unsigned* hist,
                const ChemPark& park, cudaStream_t s) {
  if (order) {
    const int nb = (d.NE + NBUCKET * SORT_ITEMS - 1) / (NBUCKET * SORT_ITEMS);
    cudaMemsetAsync(hist, 0, sizeof(unsigned) * NBUCKET, s);
    k_chem_hist<<<nb, NBUCKET, 0, s>>>(nsub, d.NE, hist);
    k_chem_scan<<<1, NBUCKET, 0, s>>>(hist);
    k_chem_scatter<<<nb, NBUCKET, 0, s>>>(nsub, d.NE, hist, order);
  }
  auto k = k_chem_source<NSP, ChemNum>;
  auto launch = [&](int grid, const ChemPark& p, int round) {
    k<<<grid, CHEM_THREADS, 0, s>>>(d, *static_cast<const ThermoDev<NSP>*>(th), tol, maxsub, nsub, order, p, round);
  };
  return (order ? 3 : 0) + chem_rounds(k, d.NE, order ? CHEM_SORTED : CHEM_UNSORTED, park, s, launch);
}

template <int NSP>
int chem_list(const Dev& d, const void* th, double tol, int maxsub, int* nsub, const int* list, const unsigned* nlist,
              const ChemPark& park, cudaStream_t s) {
  auto k = k_chem_list<NSP, ChemNum>;
  return chem_rounds(k, d.NE, CHEM_LISTED, park, s, [&](int grid, const ChemPark& p, int round) {
    k<<<grid, CHEM_THREADS, 0, s>>>(d, *static_cast<const ThermoDev<NSP>*>(th), tol, maxsub, nsub, list, nlist, p,
                                    round);
  });
}

template <int NSP>
int chem_batch(const void* th, const double* P, const double* dt, int n, double* out, int* nsub, double tol,
               int maxsub, const ChemPark& park, unsigned* errp, cudaStream_t s) {
  auto k = k_chem_batch<NSP, ChemNum>;
  return chem_rounds(k, n, CHEM_UNSORTED, park, s, [&](int grid, const ChemPark& p, int round) {
    k<<<grid, CHEM_THREADS, 0, s>>>(*static_cast<const ThermoDev<NSP>*>(th), P, dt, n, out, nsub, tol, maxsub, p,
                                    round, errp);
  });
}

#define RC_CHEM_INST(N)                                                                                         \
  template int chem_source<N>(const Dev&, const void*, double, int, int*, int*, unsigned*, const ChemPark&,     \
                              cudaStream_t);                                                                    \
  template int chem_list<N>(const Dev&, const void*, double, int, int*, const int*, const unsigned*,            \
                            const ChemPark&, cudaStream_t);                                                     \
  template int chem_batch<N>(const void*, const double*, const double*, int, double*, int*, double, int,        \
                             const ChemPark&, unsigned*, cudaStream_t);
RC_CHEM_INST(1)
RC_CHEM_INST(4)

}  // namespace rc
