// One fan-out hop of neighbour sampling over a (partly cached) CSR, as ONE kernel,
// and the sub-CSR builder that fills the cache.
//
// Reference: GetSubIndptr / GetSubIndptrWithCache + CUB scan + host read of nnz +
// CSRWise[Mask]SampleUniform[Replace]Kernel (src/cache_graph_sampling.cu:47-89,
// 222-289, 91-177, 291-380, 179-220, 382-426); CreateCacheCSR (:428-492).
//
// Here a CTA takes a tile of S seeds:
//   1. one seed per thread: cooperative map probe, row bounds from the cached
//      indptr (hit) or the host indptr over UVA (miss), picks = min(deg, k);
//   2. block scan of the picks; the tile's sum is published at once;
//   3. groups of G = 8/16/32 lanes (smallest power of two >= k) pick positions, one
//      seed each: deg <= k takes the row; otherwise each lane p < k draws
//      t_p ~ U[0, deg-k+p] with Philox4x32-10 and the group resolves Floyd's
//      subset algorithm with k shuffle+ballot steps (O(k) work, exact uniform
//      k-subset; the reference draws O(deg) numbers and uses global atomics);
//   4. look-back for the tile's offset -> sub_indptr, so no separate scan kernel and
//      no host round trip;
//   5. all threads fetch and store the picked neighbours, one each, whatever the rows'
//      lengths, and in a mini-batch claim their relabel slots.
//      k > 32: one warp per seed draws positions into a shared-memory set until k distinct
//      ones (or, for rows shorter than 2k, the deg-k to leave out) are held: O(k) draws, no
//      global atomics.  Only beyond 1024 picks per seed does it fall back to the reference's
//      reservoir on the output row.
#include <type_traits>

#include "ctx.cuh"
#include "lookback.cuh"
#include "map.cuh"
#include "relabel.cuh"

namespace shmt {

constexpr int kHopThreads = 256;
// A hop is a chain of dependent reads per edge (row bounds, neighbour, relabel slot), so resident
// threads count for more than reads in flight per thread: the third hop of 8,192 seeds x 5/10/15
// took 118 us with four edges per thread (64 registers, 4 CTAs per SM), 99 with two (5 CTAs) and 94
// with one (6 CTAs).  At 6 the 40 registers do not hold everything: 20 to 28 bytes a thread are spilled,
// and are part of the 94.
constexpr int kHopCtasPerSm = 6;
// Seeds of a tile come in steps of 8: a small hop is as long as its slowest CTA, and 1,024 seeds over
// a host graph took 20 us in 32 CTAs of 32 seeds and 16 us in 128 CTAs of 8.
constexpr int kHopSeedStep = 8;
// Relabel slots looked at first per possible edge of a hop (every row as long as the fan-out, no
// repeats): a usual hop fills a third of them.  2.0 -> 1.25 took the compact kernel behind a hop of
// 1.5 M edges from 80 to 65 us, for less of the table comes from HBM.
constexpr double kHopSlotsPerEdge = 1.25;
constexpr int kMaxSeedsPerTile = 1024;

struct HopJob {
  const void* indptr;
  const void* indices;      // host / full graph
  const void* gpu_indptr;   // compact cached CSR (nullable)
  const void* gpu_indices;
  MapView map;
  const void* seeds;
  int64_t n;
  int64_t k;
  bool indptr64, seeds64;
  bool replace;
  uint32_t rel_cap, rel_n_words, rel_tag;  // see rel_slots
  uint32_t off_lo, off_hi;
  int seeds_per_tile;
  uint32_t set_slots;     // fan-out > 32: words of the per-warp set of chosen positions (0: none)
  uint64_t rng_seed;
  void* sub_indptr;
  void* sub_indices;
  TileStates st;
  int64_t* ticket;        // tile ticket counter (starts at 0)
  int64_t* status;        // device status word
  int64_t* result;        // receives nnz
  const int64_t* n_dev;   // if set, the seed count is read here (it was produced on the device)
  // Edge ids (optional): for every sampled neighbour its position in the full `indices` array,
  // in the dtype of indptr.  A cached row's position there is gpu_edge_base[slot] + offset in row.
  void* out_eids;
  const void* gpu_edge_base;
  // Weighted sampling (optional): one positive float per edge, parallel to `indices` (and to
  // gpu_indices for the cached rows).  Always sampled by one warp per seed.
  const float* weights;
  const float* gpu_weights;
  // Fused relabel insert (multi-hop path): the kernel also claims a relabel-table slot for
  // every seed and every sampled neighbour, at its index in [seeds | neighbours], and
  // records the slot in rel_out -- the work of relabel's first kernel, done while this
  // kernel would otherwise wait on memory.  rel_slots == nullptr: off (HOP_FUSED otherwise).
  RelSlot* rel_slots;
  unsigned* rel_words;  // ids below rel_n_words take no slot, and are not recorded (see RelTable)
  void* rel_out;
  // Look-back state that the kernel itself puts back to zero (small single-hop calls): the zeroed word
  // in which its CTAs count themselves out, or nullptr.
  int64_t* clean;
  // Single-hop call with a host result: the CTA that finishes its bookkeeping last hands the
  // result words to the host, which returns while the rows are still being written.
  HostPost post;
  LaunchPad<8> pad;
};

// indptr[i] and indptr[i+1] with one load when the pair is naturally aligned (one request on
// the host link instead of two for a row that lives in host memory).  Alignment is decided on
// the address of element i, so a view that starts at an odd element (indptr[1:], an .npy
// payload at an offset that is no multiple of 16) pairs its odd rows and never issues a
// misaligned vector load.
__device__ __forceinline__ void load_bounds(const void* indptr, int is64, int64_t i, int64_t* b,
                                            int64_t* e) {
  if (is64) {
    const long long* p = reinterpret_cast<const long long*>(indptr) + i;
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
      const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(p));
      *b = v.x;
      *e = v.y;
      return;
    }
  } else {
    const int* p = reinterpret_cast<const int*>(indptr) + i;
    if ((reinterpret_cast<uintptr_t>(p) & 7) == 0) {
      const int2 v = __ldg(reinterpret_cast<const int2*>(p));
      *b = v.x;
      *e = v.y;
      return;
    }
  }
  *b = load_int(indptr, is64, i);
  *e = load_int(indptr, is64, i + 1);
}

__device__ __forceinline__ uint64_t draw_below(const Philox& rng, uint32_t seed_idx, uint32_t draw,
                                               uint32_t off_lo, uint32_t off_hi, uint64_t range) {
  const uint4 r = rng(seed_idx, draw, off_lo, off_hi);
  return bounded(r.x, r.y, range);
}

// A picked neighbour on its way through a tile: where it lies in the full or the cached index
// array, and the seed of the tile it belongs to.
struct HopEdge {
  uint64_t bits;
  __device__ __forceinline__ explicit HopEdge(uint64_t b) : bits(b) {}
  static __device__ __forceinline__ uint64_t pack(int64_t at, int seed, bool hit) {
    return (uint64_t)at | ((uint64_t)seed << 50) | ((uint64_t)hit << 63);
  }
  __device__ __forceinline__ int64_t at() const { return (int64_t)(bits & ((1ull << 50) - 1)); }
  __device__ __forceinline__ int seed() const { return (int)(bits >> 50) & ((1 << 13) - 1); }
  __device__ __forceinline__ bool hit() const { return bits >> 63; }
};
static_assert(kMaxSeedsPerTile <= 1 << 13, "a seed of the tile takes 13 bits");

// Weighted picks without replacement (Efraimidis-Spirakis 2006): every edge gets the key -log(u) / w
// (an exponential clock of rate w) and the k smallest keys win, which is sampling without
// replacement with probabilities proportional to the weights.  While a warp looks at a row, a candidate is one
// number, its key above its position, so that numbers compare as keys, equal ones by position; the warp
// holds the 32 smallest, ascending across its lanes.
using Mark = unsigned long long;
constexpr int kMarkPosBits = 32;
constexpr Mark kNoMark = ~0ull;
constexpr int kFewPicks = 4;      // taken as minima: 5,000 rows of 1,000 edges, one pick, 54 us sorted, 44 so
constexpr int kMarkBuffer = 160;  // candidates a warp collects before it sorts them: up to 31 left and 128 new

template <int N>
__device__ __forceinline__ void sort_step(Mark (&v)[N], unsigned stride, bool ascending, unsigned lane) {
  const bool low = ((lane & stride) == 0) == ascending;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const Mark other = __shfl_xor_sync(0xffffffffu, v[i], stride);
    v[i] = (v[i] < other) == low ? v[i] : other;
  }
}
// every v[i] ascending across the warp (bitonic)
template <int N>
__device__ __forceinline__ void sort_marks(Mark (&v)[N], unsigned lane) {
#pragma unroll
  for (unsigned size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (unsigned stride = size >> 1; stride > 0; stride >>= 1) sort_step<N>(v, stride, (lane & size) == 0, lane);
}
// the 32 smallest of v[i] and with[i], both ascending, into v[i]
template <int N>
__device__ __forceinline__ void merge_marks(Mark (&v)[N], const Mark* with, unsigned lane) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = min(v[i], __shfl_sync(0xffffffffu, with[i], 31 - lane));
#pragma unroll
  for (unsigned stride = 16; stride > 0; stride >>= 1) sort_step<N>(v, stride, true, lane);
}

// The k picks of a row, one per lane (0..k-1), ascending.
struct WeightedPicks {
  float key;
  int64_t pos;

  // all lanes call with the same candidate
  __device__ __forceinline__ void insert(float ck, int64_t cp, unsigned lane, int k) {
    const float left_k = __shfl_up_sync(0xffffffffu, key, 1);
    const int64_t left_p = __shfl_up_sync(0xffffffffu, pos, 1);
    if ((int)lane < k && (ck < key || (ck == key && cp < pos))) {
      const bool here = lane == 0 || left_k < ck || (left_k == ck && left_p < cp);
      key = here ? ck : left_k;
      pos = here ? cp : left_p;
    }
  }

  // The smallest marks of the edges [from, from + 128), then `step` further on, ... of `deg` with weights `w`; a
  // step's weights are loaded while the one before is looked at.  Candidates, those below the k-th smallest key
  // so far, go to `buf` and are sorted 32 to 128 at a time, the first 128 edges at once.  What bounds it is the
  // warp's chain of instructions: put in one after the other, each by a shuffle step that waits for the one
  // before, candidates cost 110 ns apiece; and with a vote and a division for every 32 edges the draws of a step
  // waited for one another, 6.6 ns an edge and warp, 4.1 now.  Calls of 5,000 rows of 200 edges: 15 picks 43 -> 30 us,
  // 32 picks 58 -> 31, of 1,000 edges 77 -> 59 and 102 -> 65; one row of 10,000: 38 -> 28, 100 of 100,000: 760 -> 540.
  static __device__ __forceinline__ Mark scan_marks(const float* w, unsigned from, unsigned step, unsigned deg,
                                                    unsigned lane, int k, const Philox& rng, uint32_t seed_idx,
                                                    uint32_t counter0, uint32_t off_lo, uint32_t off_hi, Mark* buf) {
    constexpr int U = 4;
    const unsigned full = 0xffffffffu;
    const float tiny = 1.17549435e-38f, most = 3.40282347e+38f;  // smallest weight, largest key
    float next[U];
#pragma unroll
    for (int u = 0; u < U; ++u) next[u] = from + 32 * u + lane < deg ? __ldg(w + from + 32 * u + lane) : 1.0f;
    Mark best[1] = {kNoMark};
    float thr = __int_as_float(0x7f800000), above = thr;  // the bound, and one that roundings do not reach
    int held = 0;
    for (unsigned p0 = from; p0 < deg; p0 += step) {
      float cur[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        cur[u] = next[u];
        const unsigned ahead = p0 + step + 32 * u + lane;
        if (ahead < deg) next[u] = __ldg(w + ahead);
      }
      // the key is clock / weight; whether any may lie below the bound is seen without dividing, and at once
      float clock[U];
      bool maybe = false;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned at = p0 + 32 * u + lane;
        const uint4 r = rng(seed_idx, counter0 + at, off_lo, off_hi);
        const float x = ((float)(r.x >> 8) + 1.0f) * (1.0f / 16777216.0f);  // (0, 1]
        clock[u] = -__logf(x);
        cur[u] = fmaxf(cur[u], tiny);  // a weight that is not positive counts as the smallest; its edge can still be picked
        maybe = maybe || (at < deg && clock[u] <= above * cur[u]);
      }
      if (__any_sync(full, maybe)) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned at = p0 + 32 * u + lane;
          const float mine = fabsf(fminf(clock[u] / cur[u], most));  // no negative zero
          const bool cand = at < deg && mine < thr;
          const unsigned votes = __ballot_sync(full, cand);
          if (cand) buf[held + __popc(votes & ((1u << lane) - 1u))] = ((Mark)__float_as_uint(mine) << kMarkPosBits) | at;
          held += __popc(votes);
        }
      }
      const bool last = p0 + step >= deg;
      while (held >= 32 || (last && held > 0)) {
        __syncwarp();
        const int n = min(held, 128);
        held -= n;
        if (k <= kFewPicks) {  // the k smallest one after the other
          Mark v[5] = {best[0]}, kept = kNoMark;
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u + 1] = 32 * u + (int)lane < n ? buf[held + 32 * u + lane] : kNoMark;
          for (int t = 0; t < k; ++t) {
            Mark least = v[0];
#pragma unroll
            for (int u = 1; u < 5; ++u) least = min(least, v[u]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) least = min(least, __shfl_xor_sync(full, least, o));
            if ((int)lane == t) kept = least;
#pragma unroll
            for (int u = 0; u < 5; ++u)
              if (v[u] == least) v[u] = kNoMark;
          }
          best[0] = kept;
        } else if (n <= 32) {
          Mark v[1] = {(int)lane < n ? buf[held + lane] : kNoMark};
          sort_marks<1>(v, lane);
          merge_marks<1>(best, v, lane);
        } else {
          Mark v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = 32 * u + (int)lane < n ? buf[held + 32 * u + lane] : kNoMark;
          sort_marks<4>(v, lane);
          Mark two[2] = {v[0], v[1]};
          merge_marks<2>(two, v + 2, lane);
          Mark one[1] = {two[0]};
          merge_marks<1>(one, two + 1, lane);
          merge_marks<1>(best, one, lane);
        }
        const unsigned bits = (unsigned)(__shfl_sync(full, best[0], k - 1) >> kMarkPosBits);
        thr = __uint_as_float(min(bits, 0x7f800000u));
        above = thr * 1.0001f;
        __syncwarp();
      }
    }
    return best[0];
  }

  // The same of a whole row (or this warp's share of it).  `key` and `pos` are those of no pick where there are
  // fewer than k.  Rows of more than 2^31 edges are looked at piece by piece.
  __device__ __forceinline__ void scan(const float* w, unsigned from, unsigned step, int64_t deg, unsigned lane, int k,
                                       const Philox& rng, uint32_t seed_idx, uint32_t off_lo, uint32_t off_hi,
                                       Mark* buf) {
    constexpr int64_t kPiece = (int64_t)1 << 31;
    for (int64_t p0 = 0; p0 < deg; p0 += kPiece) {
      const Mark m = scan_marks(w + p0, from, step, (unsigned)min(deg - p0, kPiece), lane, k, rng, seed_idx, (uint32_t)p0, off_lo,
                                off_hi, buf);
      const float mk = m == kNoMark ? __int_as_float(0x7f800000) : __uint_as_float((unsigned)(m >> kMarkPosBits));
      const int64_t mp = m == kNoMark ? -1 : p0 + (int64_t)(unsigned)m;
      if (p0 == 0) {
        key = mk;
        pos = mp;
        continue;
      }
      for (int t = 0; t < k; ++t) {
        const float ck = __shfl_sync(0xffffffffu, mk, t);
        const int64_t cp = __shfl_sync(0xffffffffu, mp, t);
        if (cp >= 0) insert(ck, cp, lane, k);
      }
    }
  }
};

// Which rows of a tile the warps of the CTA share (a row's edges dealt out 128 at a time, the warps' picks
// then ranked against one another), and which ones a warp takes alone: a hop is as long as its slowest
// tile.  Alone rows run beside one another, shared rows one after the other, and a shared row is less
// than an eighth as long: each warp still sorts its own candidates.  So the longest rows are shared, as
// many of them as make the tile's estimate smallest.
// Shorter rows are never shared (lines at 256 and 512: the same within 1 %, and 2 % behind on hops of 4,000 seeds).
constexpr int64_t kWeightedLongRow = 1024;
// Times in edges looked at (4 ns): the first sort is worth 170; behind the first 128 edges about k * ln(edges / 128)
// candidates are collected, and sorted 32 at a time for 100.
__device__ __forceinline__ float weighted_cost(float edges, float k) {
  if (edges <= k) return k;
  return edges + 170.0f + (edges > 128.0f ? 100.0f + 3.0f * k * __logf(edges / 128.0f) : 0.0f);
}
constexpr float kWeightedShareCost = 200.0f;  // barriers, and the ranking

// HOP_FUSED: a hop of a mini-batch, which also claims relabel slots.  HOP_SINGLE: a call of its own.  Kernels
// apart, because the claims' code and registers cost a small call 0.7 of 24 us though it never runs it.  HOP_EARLY: a
// weighted call whose count the host waits for (see step 3).
// HOP_TINY: a call of its own for few seeds.  Every CTA looks all seeds up and adds up all picks itself: no ticket, no
// look-back, nobody counts anybody out, and the count is on its way to the host before a position is picked.  100
// seeds on the GPU 23.6 us a call, 19.5 so; 1,024 24.0 and 22.4.
enum : int { HOP_FUSED = 0, HOP_SINGLE = 1, HOP_EARLY = 2, HOP_TINY = 3 };
// Beyond a few seeds a thread the CTAs' repeated lookups cost what the look-back does.  Over a host graph each CTA reads
// all row bounds across the link: 50 seeds 25.0 us the other way and 22.7 so, 100 seeds 26.0 and 26.6, 256 seeds 26.9
// and 51.7.
constexpr int64_t kTinySeeds = 4 * kHopThreads, kTinyHostSeeds = 64;

// Reductions on one address are served one after the other, 1.15 ns each, so the word of a node that many edges lead to
// must not get one for every edge.  A CTA of a mini-batch's hop keeps the ids whose words it has lowered, the last
// at each place: an id below 2^25 times an odd number, modulo 2^25, has its place in the upper 10 bits, and the lower 15 tell
// ids of one place apart; below them, in the entry, the index within the tile.  A neighbour whose id is there with a
// smaller index leaves the word alone: whoever made the entry lowers it as far, or has left that to a smaller index still.
// 8,192 seeds 5/10/15 on 10 M nodes, int64 ids: a tenth of all edges to one node 964 us without, 394 so (third hop 809 and 142;
// hashed slots 560), neighbours by rank^-1.1 236 and 145 (slots 188), drawn evenly 344 both; 1,024 seeds 221 and 133, 106 and 107,
// 127 and 129.  With 8-byte entries, and lanes that meet looked for in every step, not in the first alone, 344 was 373.
constexpr int kLoweredTagBits = 15, kLoweredEntries = (int)(kRelMaxWords >> kLoweredTagBits);
constexpr unsigned kLoweredLocal = (1u << (32 - kLoweredTagBits)) - 1u;
// To look for lanes that meet costs a hop 0.5 us, so hops of fewer possible edges do without: with a line at 0, 2^15, 2^16 and
// 2^17, 50 seeds 64.5, 66.7, 66.0 and 66.0 us (62.2 and 66.0 without any of this, the first on another box), 1,024
// seeds 125.8, 127, 126.9 and 126.0 (124.3, 124.7), 1,024 of them on 10 M nodes with a tenth of all edges to one 127, 128, 134
// and 134 (220).
constexpr int64_t kCrowdedEdges = 1 << 16;
// What a kernel may take beside its arrays of fixed size, at most 8 KB, without asking for more.
constexpr size_t kPlainHopSmem = 40 << 10;

template <typename IxT, int G, int MODE>
__global__ void __launch_bounds__(kHopThreads, G < 32 ? kHopCtasPerSm : 4) sample_hop_kernel(const HopJob job) {
  extern __shared__ __align__(16) unsigned char s_dyn[];  // hop_smem_bytes()
  __shared__ int64_t warp_sums[32];
  __shared__ int64_t s_total;
  __shared__ LookbackShared s_look;
  __shared__ int s_tile;
  __shared__ int64_t s_prefix, s_end;  // HOP_TINY
  __shared__ unsigned s_lowered[MODE == HOP_FUSED ? kLoweredEntries : 1];

  pdl_launch_next();
  if (MODE == HOP_FUSED)  // the barriers of the pick counts' scan lie before its first use
    for (int q = (int)threadIdx.x; q < kLoweredEntries; q += kHopThreads) s_lowered[q] = ~0u;
  pdl_wait();
  const unsigned full = 0xffffffffu;
  const unsigned tid = threadIdx.x, lane = tid & 31;
  const int S = job.seeds_per_tile;
  int64_t* s_begin = reinterpret_cast<int64_t*>(s_dyn);
  int64_t* s_deg = s_begin + S;
  int64_t* s_off = s_deg + S;
  int64_t* s_eshift = s_off + S;  // edge id = position read from + this (edge ids only)
  uint8_t* s_hit = reinterpret_cast<uint8_t*>(s_eshift + S);
  // one of the two behind them: the picked neighbours of the tile in output order (k <= 32), or per
  // warp a set of chosen positions (job.set_slots words)
  uint64_t* s_list = reinterpret_cast<uint64_t*>(s_hit + S);
  uint32_t* s_sets = reinterpret_cast<uint32_t*>(s_hit + S);
  const int64_t n = job.n_dev ? *job.n_dev : job.n;
  const int64_t n_tiles = (n + S - 1) / S;
  if (blockIdx.x >= n_tiles) {  // the grid is sized for the largest n the caller allows
    if (n == 0 && blockIdx.x == 0 && tid < 32) {
      if (tid == 0) {
        store_int(job.sub_indptr, job.indptr64, 0, 0);
        st_relaxed64(job.result, 0);
        __threadfence();
      }
      __syncwarp();
      post_to_host(job.post);
    }
    return;
  }
  constexpr bool kFused = MODE == HOP_FUSED, kEarly = MODE == HOP_EARLY, kTiny = MODE == HOP_TINY;
  const int tile = kTiny ? (int)blockIdx.x : take_tile(job.ticket, &s_tile);  // as many CTAs as tiles are left
  if (!kFused && job.clean && tile == 0 && tid == 0) st_relaxed64(job.status, DEV_OK);  // it reports on this call only
  const int64_t first = (int64_t)tile * S;
  const int rows = (int)min((int64_t)S, n - first);
  const int64_t k = job.k;

  // ---- 1. row bounds and pick counts, one seed per thread
  if (kTiny) {  // of all seeds, a few in a row per thread; this CTA's are kept
    auto add_up = [&](auto most) -> int64_t {
      constexpr int kMost = decltype(most)::value;
      const int per = kMost == 1 ? 1 : (int)((n + kHopThreads - 1) / kHopThreads);
      int64_t row[kMost], slot[kMost], b[kMost], e[kMost];
#pragma unroll
      for (int q = 0; q < kMost; ++q) {
        const int i = (int)tid * per + q;
        row[q] = q < per && i < n ? load_int(job.seeds, job.seeds64, i) : kEmptyKey;
      }
#pragma unroll
      for (int q = 0; q < kMost; ++q) {
        if (q >= per) break;
        const bool valid = (int64_t)tid * per + q < n;
        slot[q] = -1;
        if (job.map.slots) slot[q] = warp_find(job.map, row[q], valid);
        b[q] = e[q] = 0;
        if (valid) {
          if (slot[q] >= 0)
            load_bounds(job.gpu_indptr, job.indptr64, slot[q], &b[q], &e[q]);
          else
            load_bounds(job.indptr, job.indptr64, row[q], &b[q], &e[q]);
        }
      }
      auto picks = [&](int q) -> int64_t {
        if (q >= per || (int64_t)tid * per + q >= n) return 0;
        const int64_t deg = e[q] - b[q];
        return job.replace ? (deg > 0 ? k : 0) : (deg < k ? deg : k);
      };
      int64_t sum = 0;
#pragma unroll
      for (int q = 0; q < kMost; ++q) sum += picks(q);
      int64_t run = block_exclusive_scan(sum, warp_sums, &s_total);
#pragma unroll
      for (int q = 0; q < kMost; ++q) {
        const int i = (int)tid * per + q, j = i - (int)first;
        if (q < per && j >= 0 && j < rows) {
          s_begin[j] = b[q];
          s_deg[j] = e[q] - b[q];
          s_hit[j] = slot[q] >= 0;
          s_off[j] = run;
          if (job.out_eids) s_eshift[j] = slot[q] >= 0 ? load_int(job.gpu_edge_base, job.indptr64, slot[q]) - b[q] : 0;
          store_int(job.sub_indptr, job.indptr64, i, run);
          if (j == rows - 1) s_end = run + picks(q);
        }
        run += picks(q);
      }
      return s_total;
    };
    const int64_t total = n <= kHopThreads ? add_up(std::integral_constant<int, 1>{})
                                           : add_up(std::integral_constant<int, (int)(kTinySeeds / kHopThreads)>{});
    if (tile == 0 && tid < 32) {
      if (tid == 0) {
        store_int(job.sub_indptr, job.indptr64, n, total);
        st_relaxed64(job.status, DEV_OK);
        st_relaxed64(job.result, total);
      }
      post_result(job.post, total);
    }
    __syncthreads();
    const int64_t prefix = s_off[0];
    __syncthreads();
    for (int j = (int)tid; j < rows; j += kHopThreads) s_off[j] -= prefix;
    if (tid == 0) {
      s_prefix = prefix;
      s_total = s_end - prefix;
    }
    __syncthreads();
  }
  for (int j0 = (int)(tid & ~31u); !kTiny && j0 < S; j0 += kHopThreads) {
    const int j = j0 + (int)lane;
    const bool valid = j < rows;
    const int64_t row = valid ? load_int(job.seeds, job.seeds64, first + j) : kEmptyKey;
    int64_t slot = -1;
    if (job.map.slots) slot = warp_find(job.map, row, valid);
    int64_t b = 0, e = 0;
    if (valid) {
      if (slot >= 0)
        load_bounds(job.gpu_indptr, job.indptr64, slot, &b, &e);
      else
        load_bounds(job.indptr, job.indptr64, row, &b, &e);
    }
    const int64_t deg = e - b;
    if (job.out_eids && j < S)
      s_eshift[j] = (valid && slot >= 0) ? load_int(job.gpu_edge_base, job.indptr64, slot) - b : 0;
    if (j < S) {
      s_begin[j] = b;
      s_deg[j] = deg;
      s_hit[j] = slot >= 0;
      s_off[j] = !valid ? 0 : (job.replace ? (deg > 0 ? k : 0) : (deg < k ? deg : k));
    }
  }
  __syncthreads();

  // ---- 2. offsets inside the tile.  The tile's sum goes out now: the tiles behind it then never
  // wait for the neighbour loads and slot claims below.
  if (!kTiny) {
    const int ch = (S + kHopThreads - 1) / kHopThreads;  // seeds per thread, 1..4
    int64_t c[kMaxSeedsPerTile / kHopThreads];
    int64_t sum = 0;
#pragma unroll
    for (int q = 0; q < kMaxSeedsPerTile / kHopThreads; ++q) {
      const int j = (int)tid * ch + q;
      c[q] = (q < ch && j < S) ? s_off[j] : 0;
      sum += c[q];
    }
    int64_t run = block_exclusive_scan(sum, warp_sums, &s_total);
    if (tid == 0) lookback_publish(job.st, tile, s_total);
#pragma unroll
    for (int q = 0; q < kMaxSeedsPerTile / kHopThreads; ++q) {
      const int j = (int)tid * ch + q;
      if (q < ch && j < S) s_off[j] = run;
      run += c[q];
    }
    __syncthreads();
  }

  constexpr int kGroups = kHopThreads / G;
  const unsigned gl = tid & (G - 1);
  const unsigned gshift = lane & ~(unsigned)(G - 1);  // first lane of my group within the warp
  const unsigned gmask = G == 32 ? full : (((1u << G) - 1u) << gshift);
  const int group = (int)(tid / G);
  const Philox rng(job.rng_seed);
  IxT* out_all = static_cast<IxT*>(job.sub_indices);
  const bool listed = G < 32 || (k <= G && !(job.weights && job.replace));  // a smaller group is only launched for such calls
  const double most = (double)n * (double)(1 + k);  // ids of this hop, were every row that long
  const RelRange range{job.rel_slots,
                       kFused ? relabel_near(most, relabel_slots_per_id(most, kHopSlotsPerEdge), job.rel_cap) : 0u,
                       job.rel_cap};
  const bool crowds = n * k >= kCrowdedEdges;
  // The word of node `id`, unless this CTA has lowered it as far (s_lowered).  `local`, the index within the tile as
  // far as it can be held, goes up with `i`.
  auto lower = [&](unsigned id, unsigned i, unsigned local, bool crowd) {
    const unsigned mixed = id * 0x9E3779B1u & (kRelMaxWords - 1);
    volatile unsigned* last = s_lowered + (mixed >> kLoweredTagBits);
    const unsigned mine = mixed << (32 - kLoweredTagBits) | local;
    unsigned seen = *last;
    if (seen < mine && (seen ^ mine) <= kLoweredLocal) return;
    *last = mine;
    unsigned* word = job.rel_words + id;
    if (crowd) {  // nothing is known yet: lanes that meet here leave it to the lowest, which looks first
      seen = *last;  // of several lanes' stores one
      if (seen < mine && (seen ^ mine) <= kLoweredLocal) return;
      const unsigned together = __activemask();
      if (__any_sync(together, seen != mine)) {
        const unsigned same = __match_any_sync(together, id);
        if (__shfl_sync(same, i, __ffs(same) - 1) < i) return;
        if (same & (same - 1u) && __ldcg(word) <= job.rel_tag + i) return;
      }
    }
    atomicMin(word, job.rel_tag + i);
  };
  // the id at index i of [seeds | neighbours]: its slot, for the later relabel passes
  auto enter = [&](int64_t i, IxT id, int64_t local, bool crowd) {
    if ((uint64_t)(long long)id < job.rel_n_words) {
      if (local < rows && job.n_dev)  // the distinct ids of the hop before
        atomicMin(job.rel_words + id, job.rel_tag + (unsigned)i);
      else
        lower((unsigned)id, (unsigned)i, (unsigned)min(local, (int64_t)kLoweredLocal), crowd);
      return;
    }
    bool maybe_first;
    const uint32_t at = relabel_enter<false>(range, (long long)id, (unsigned)i, job.status, &maybe_first);
    store_int(job.rel_out, sizeof(IxT) == 8, i, relabel_pack(at, maybe_first, sizeof(IxT) == 8));
  };

  // the tile's place in the output, and what the host waits for
  auto place = [&]() -> int64_t {
    const int64_t prefix = lookback_block(job.st, tile, s_total, &s_look, job.status);
    for (int j = (int)tid; j < rows; j += kHopThreads)
      store_int(job.sub_indptr, job.indptr64, first + j, prefix + s_off[j]);
    if (tile == n_tiles - 1 && tid == 0) {
      store_int(job.sub_indptr, job.indptr64, n, prefix + s_total);
      st_relaxed64(job.result, prefix + s_total);
    }
    if (!kFused && job.post.host) {  // uniform over the grid
      __syncthreads();
      if (!job.clean && tid < 32) post_when_last(job.post, n_tiles);
    }
    if (!kFused && job.clean) {  // uniform as well; all look-backs of this CTA are over
      if (!job.post.host) __syncthreads();
      if (tid < 32 && last_to_finish(job.clean, n_tiles)) {
        for (int64_t t = lane; t < n_tiles; t += 32) st_desc(job.st.d + t, 0, 0);
        if (lane == 0) {
          st_relaxed64(job.ticket, 0);
          st_relaxed64(job.clean, 0);
        }
        // only now: the host may queue the state's next user in another stream as soon as it has the post
        post_to_host(job.post);
      }
    }
    return prefix;
  };

  // Picking by weight takes long, and a host that waits for the count need not wait for it, so the
  // tile takes its place first (8 rows of 1,000 edges, 15 picks each: 46.6 us a call, 31.2 so).  Both orders in one
  // kernel cost the other one: a weighted mini-batch of 1,000 seeds 130 us for 125.
  const int64_t placed = kEarly ? place() : (kTiny ? s_prefix : 0);

  // ---- 3. (k <= 32) positions of the picked neighbours, a group of lanes per seed, into a list in
  // output order.  Arithmetic and shuffles only: the memory work is left to step 5, where all
  // threads of the tile share it evenly whatever the rows' lengths.
  if (G == 32 && listed && job.weights && k > 0) {
    __shared__ float s_key[G == 32 ? kHopThreads : 1];
    __shared__ int64_t s_pos[G == 32 ? kHopThreads : 1];
    __shared__ unsigned long long s_cut;
    const float none = __int_as_float(0x7f800000);
    Mark* marks = reinterpret_cast<Mark*>(s_list + S * 32) + group * kMarkBuffer;  // behind the list
    auto weights_of = [&](int j) { return (s_hit[j] ? job.gpu_weights : job.weights) + s_begin[j]; };
    auto list = [&](int j, int at, int64_t pos) {
      s_list[s_off[j] + at] = HopEdge::pack(s_begin[j] + pos, j, s_hit[j]);
    };
    // rows in falling order of length (then by place): those ahead of row `cut` are shared.  A single long
    // row always is.
    int cut = -1;
    int64_t cut_deg = kWeightedLongRow;
    const int64_t my_deg = (int)tid < rows ? s_deg[tid] : -1;  // thread `rows` stands behind the last row
    const int n_long = __syncthreads_count(my_deg > kWeightedLongRow);
    if (n_long == 1) cut = 0;
    if (n_long > 1) {
      const float fk = (float)k;
      if (tid == 0) s_cut = ~0ull;
      if ((int)tid < rows) {
        s_key[tid] = weighted_cost((float)my_deg, fk);
        reinterpret_cast<float*>(s_pos)[tid] = weighted_cost((float)my_deg / kGroups, fk) + kWeightedShareCost;
      }
      __syncthreads();
      if ((int)tid <= rows) {
        float shared = 0.0f, alone = 0.0f;
        bool allowed = true;
        for (int j = 0; j < rows; ++j) {
          if (s_deg[j] > my_deg || (s_deg[j] == my_deg && j < (int)tid)) {
            shared += reinterpret_cast<const float*>(s_pos)[j];
            allowed = allowed && s_deg[j] > kWeightedLongRow;
          } else {
            alone += s_key[j];
          }
        }
        const float mine = (int)tid < rows ? s_key[tid] : 0.0f;
        const float estimate = shared + fmaxf(mine, alone / kGroups);
        if (allowed) atomicMin(&s_cut, ((unsigned long long)__float_as_uint(estimate) << 32) | tid);
      }
      __syncthreads();
      cut = (int)(s_cut & 0xFFFFFFFFull);
      cut_deg = cut < rows ? s_deg[cut] : -1;
    }
    auto is_shared = [&](int j) {  // the same on every thread
      return cut >= 0 && (s_deg[j] > cut_deg || (s_deg[j] == cut_deg && j < cut));
    };
    for (int j = group; j < rows; j += kGroups) {
      const int64_t deg = s_deg[j];
      if (deg <= k) {
        if ((int64_t)gl < deg) list(j, (int)gl, gl);
      } else if (!is_shared(j)) {
        WeightedPicks best{none, -1};
        best.scan(weights_of(j), 0, 128, deg, gl, (int)k, rng, (uint32_t)(first + j), job.off_lo, job.off_hi, marks);
        if ((int64_t)gl < k) list(j, (int)gl, best.pos);
      }
    }
    for (int j = 0; cut >= 0 && j < rows; ++j) {
      if (!is_shared(j)) continue;
      WeightedPicks best{none, -1};
      best.scan(weights_of(j), group * 128, kGroups * 128, s_deg[j], gl, (int)k, rng, (uint32_t)(first + j), job.off_lo,
                job.off_hi, marks);
      __syncthreads();  // the row before has been ranked (and the estimates read)
      s_key[tid] = best.key;
      s_pos[tid] = best.pos;
      __syncthreads();
      // a pick's place is the number of picks ahead of it, found in each warp's ascending list; one that
      // its warp has not filled has k ahead of it
      int ahead[kGroups] = {0}, rank = 0;
      for (int step = 1 << (31 - __clz((int)k)); step > 0; step >>= 1) {
#pragma unroll
        for (int w = 0; w < kGroups; ++w) {
          const int at = w * 32 + min(ahead[w] + step, (int)k) - 1;
          const float ck = s_key[at];
          const bool less = ck < best.key || (ck == best.key && s_pos[at] < best.pos);
          if (less && ahead[w] + step <= (int)k) ahead[w] += step;
        }
      }
#pragma unroll
      for (int w = 0; w < kGroups; ++w) rank += ahead[w];
      if ((int64_t)gl < k && rank < (int)k) list(j, rank, best.pos);
    }
    __syncthreads();
  } else if (listed) {
    for (int j0 = 0; j0 < rows; j0 += kGroups) {
      const int j = j0 + group;
      const bool active = j < rows;
      const int64_t deg = active ? s_deg[j] : 0;
      const uint32_t seed_idx = (uint32_t)(first + j);
      int64_t pos = -1;
      if (job.replace) {
        if (deg > 0 && (int64_t)gl < k)
          pos = (int64_t)draw_below(rng, seed_idx, gl, job.off_lo, job.off_hi, (uint64_t)deg);
      } else {
        if (active && deg <= k && (int64_t)gl < deg) pos = gl;
        const bool pick = active && deg > k;
        // Floyd: step p inserts t_p unless already chosen, then inserts deg-k+p instead
        if (__any_sync(full, pick)) {
          const int64_t top = deg - k + (int64_t)gl;  // largest position step gl may choose
          int64_t t = -1;
          if (pick && (int64_t)gl < k)
            t = (int64_t)draw_below(rng, seed_idx, gl, job.off_lo, job.off_hi, (uint64_t)top + 1);
          int64_t res = -1;
          for (int p = 0; p < (int)k; ++p) {
            const int64_t cand = __shfl_sync(full, t, p, G);
            const bool clash = pick && (int)gl < p && res == cand;
            const unsigned votes = __ballot_sync(full, clash) & gmask;
            if ((int)gl == p) res = votes ? top : cand;
          }
          if (pick && (int64_t)gl < k) pos = res;
        }
      }
      if (pos >= 0) s_list[s_off[j] + gl] = HopEdge::pack(s_begin[j] + pos, j, s_hit[j]);
    }
    __syncthreads();
  }

  // ---- 4. the tile's place in the output.  The first neighbours are fetched ahead of the look-back,
  // so that the two waits overlap.
  const int lead = kFused ? rows : 0;  // the seeds come first: they are relabelled too
  const int n_items = listed ? lead + (int)s_total : 0;
  auto fetch = [&](int e) -> IxT {
    if (e >= n_items) return IxT(0);
    if (e < lead) return (IxT)load_int(job.seeds, job.seeds64, first + e);
    const HopEdge x(s_list[e - lead]);
    return __ldg(static_cast<const IxT*>(x.hit() ? job.gpu_indices : job.indices) + x.at());
  };
  IxT next = fetch((int)tid);
  const int64_t prefix = kEarly || kTiny ? placed : place();

  // ---- 5. output and relabel slots, one list element per thread and step
  if (listed) {
    for (int e = (int)tid; e < n_items; e += kHopThreads) {
      const IxT v = next;
      next = fetch(e + kHopThreads);
      int64_t i = first + e;  // index in [seeds | neighbours]
      if (e >= lead) {
        const int64_t o = prefix + (e - lead);
        i = n + o;
        out_all[o] = v;
        if (job.out_eids) {
          const HopEdge x(s_list[e - lead]);
          store_int(job.out_eids, job.indptr64, o, x.at() + s_eshift[x.seed()]);
        }
      }
      if (kFused) enter(i, v, e, crowds && e < lead + kHopThreads);
    }
    return;
  }
  if (kFused)
    for (int j = (int)tid; j < rows; j += kHopThreads)
      enter(first + j, (IxT)load_int(job.seeds, job.seeds64, first + j), j, crowds);

  // k > 32, or weighted with replacement (G == 32): one warp per seed
  const uint32_t set_slots = job.set_slots;
  uint32_t* set = s_sets + (size_t)(tid >> 5) * set_slots;
  for (int j0 = 0; j0 < rows; j0 += kGroups) {
    const int j = j0 + group;
    const bool active = j < rows;
    const int64_t deg = active ? s_deg[j] : 0;
    const IxT* in = nullptr;
    int64_t out_at = 0;
    if (active) {
      in = static_cast<const IxT*>(s_hit[j] ? job.gpu_indices : job.indices) + s_begin[j];
      out_at = prefix + s_off[j];
    }
    const uint32_t seed_idx = (uint32_t)(first + j);
    // one output element: the neighbour at `pos` of the row goes to slot `o` of the output
    auto emit = [&](int64_t o, int64_t pos) {
      const IxT val = __ldg(in + pos);
      out_all[o] = val;
      if (job.out_eids) store_int(job.out_eids, job.indptr64, o, s_begin[j] + pos + s_eshift[j]);
      if (kFused) enter(n + o, val, rows + (o - prefix), false);
    };
    if (job.weights && deg > 0 && job.replace) {
      const float* w = (s_hit[j] ? job.gpu_weights : job.weights) + s_begin[j];
      const float tiny = 1.17549435e-38f;  // a weight that is not positive counts as the smallest one
      {
        // k independent draws proportional to the weights: the row's total, then for 32 draws at
        // a time a second walk that finds where each draw's share of the total falls
        double sum = 0.0;
        for (int64_t p = gl; p < deg; p += 32) sum += (double)fmaxf(__ldg(w + p), tiny);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
        for (int64_t d0 = 0; d0 < k; d0 += 32) {
          const bool mine = d0 + gl < k;
          const uint4 r = rng(seed_idx, (uint32_t)(d0 + gl), job.off_lo, job.off_hi);
          const double target = ((double)r.x + 0.5) * (1.0 / 4294967296.0) * sum;
          int64_t found = -1;
          double base = 0.0;
          for (int64_t p0 = 0; p0 < deg; p0 += 32) {
            const int64_t pos = p0 + gl;
            double inc = pos < deg ? (double)fmaxf(__ldg(w + pos), tiny) : 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const double up = __shfl_up_sync(full, inc, o);
              if (gl >= (unsigned)o) inc += up;
            }
            const double chunk_end = base + __shfl_sync(full, inc, 31);
            const bool here = mine && found < 0 && target < chunk_end;
            if (__any_sync(full, here)) {
              for (int q = 0; q < 32; ++q) {
                const double upto = base + __shfl_sync(full, inc, q);
                if (here && found < 0 && target < upto && p0 + q < deg) found = p0 + q;
              }
            }
            base = chunk_end;
          }
          if (mine) emit(out_at + d0 + gl, found >= 0 ? found : deg - 1);
        }
      }
      continue;
    }
    if (job.replace) {
      if (deg <= 0) continue;
      auto drawn = [&](int64_t p) {
        return (int64_t)draw_below(rng, seed_idx, (uint32_t)p, job.off_lo, job.off_hi, (uint64_t)deg);
      };
      // The plain hop has a short loop of its own, not unrolled: 200,000 seeds with 200 draws take 185 us (two draws a
      // step 184, but 33 to 40 draws 107 for 84).
      if (!kFused && !job.out_eids) {
#pragma unroll 1
        for (int64_t p = gl; p < k; p += 32) out_all[out_at + p] = __ldg(in + drawn(p));
      } else {
        for (int64_t p = gl; p < k; p += 32) emit(out_at + p, drawn(p));
      }
      continue;
    }
    if (deg <= k) {
      for (int64_t p = gl; p < deg; p += 32) emit(out_at + p, p);
      continue;
    }
    if (set_slots == 0 || deg >= 0xFFFFFFFFll) {
      // fan-outs beyond the shared-memory set (or rows of 2^32 neighbours): the reservoir on the
      // output row, O(deg) draws (src/cache_graph_sampling.cu:329-345)
      IxT* out = out_all + out_at;
      for (int64_t p = gl; p < k; p += 32) out[p] = (IxT)p;
      __syncwarp();
      for (int64_t q = k + gl; q < deg; q += 32) {
        const uint64_t r = draw_below(rng, seed_idx, (uint32_t)q, job.off_lo, job.off_hi, (uint64_t)q + 1);
        if (r < (uint64_t)k) atomicMax(out + r, (IxT)q);
      }
      __syncwarp();
      __threadfence_block();
      for (int64_t p = gl; p < k; p += 32) {
        const IxT pos = *reinterpret_cast<volatile IxT*>(out + p);
        emit(out_at + p, (int64_t)pos);
      }
      continue;
    }
    // A uniform k-subset in O(k) draws, all in shared memory: positions are drawn independently
    // and kept if new, until m distinct ones are held (any rule that treats all positions alike
    // yields every subset with the same probability).  m = k when the row is at least twice the
    // fan-out; otherwise the deg - k positions to LEAVE OUT are drawn, so at most half of the
    // draws are ever rejected.  The set is an open-addressing table of 2^x >= 2k words per warp.
    const bool complement = deg < 2 * k;
    const uint32_t m = (uint32_t)(complement ? deg - k : k);
    const uint32_t smask = set_slots - 1;
    for (uint32_t q = gl; q < set_slots; q += 32) set[q] = 0xFFFFFFFFu;
    __syncwarp();
    uint32_t held = 0, draws = 0;
    // a draw is rejected with probability below 1/2, so a few rounds suffice; the cap only makes
    // the loop provably finite
    for (int round = 0; held < m && round < 256 + (int)(m >> 2); ++round) {
      const bool mine = held + gl < m;
      bool kept = false;
      if (mine) {
        const uint32_t pos = (uint32_t)draw_below(rng, seed_idx, draws + gl, job.off_lo, job.off_hi, (uint64_t)deg);
        uint32_t at = (pos * 0x9E3779B1u) & smask;
        while (true) {
          const uint32_t old = atomicCAS(set + at, 0xFFFFFFFFu, pos);
          if (old == 0xFFFFFFFFu) { kept = true; break; }
          if (old == pos) break;
          at = (at + 1) & smask;
        }
      }
      held += (uint32_t)__popc(__ballot_sync(full, kept));
      draws += 32;
    }
    __syncwarp();
    if (held < m && gl == 0) {
      // never reached in practice: complete the set with the lowest positions not in it
      for (uint32_t pos = 0; held < m && pos < (uint32_t)deg; ++pos) {
        uint32_t at = (pos * 0x9E3779B1u) & smask;
        while (set[at] != 0xFFFFFFFFu && set[at] != pos) at = (at + 1) & smask;
        if (set[at] == 0xFFFFFFFFu) {
          set[at] = pos;
          ++held;
        }
      }
    }
    __syncwarp();
    if (!complement) {
      // the chosen positions, in table order
      uint32_t done = 0;
      for (uint32_t q0 = 0; q0 < set_slots; q0 += 32) {
        const uint32_t pos = set[q0 + gl];
        const unsigned has = __ballot_sync(full, pos != 0xFFFFFFFFu);
        if (pos != 0xFFFFFFFFu) emit(out_at + done + __popc(has & ((1u << gl) - 1u)), (int64_t)pos);
        done += (uint32_t)__popc(has);
      }
    } else {
      // every position that was not drawn, in row order
      uint32_t done = 0;
      for (int64_t p0 = 0; p0 < deg; p0 += 32) {
        const int64_t pos = p0 + gl;
        bool keep = pos < deg;
        if (keep) {
          uint32_t at = ((uint32_t)pos * 0x9E3779B1u) & smask;
          while (true) {
            const uint32_t cur = set[at];
            if (cur == 0xFFFFFFFFu) break;
            if (cur == (uint32_t)pos) { keep = false; break; }
            at = (at + 1) & smask;
          }
        }
        const unsigned has = __ballot_sync(full, keep);
        if (keep) emit(out_at + done + __popc(has & ((1u << gl) - 1u)), pos);
        done += (uint32_t)__popc(has);
      }
    }
    __syncwarp();  // the set is cleared for the next seed only after every lane has read it
  }
}

// ---- sub-CSR ------------------------------------------------------------------

__global__ void subcsr_degree_kernel(const void* __restrict__ indptr, int indptr64,
                                     const void* __restrict__ seeds, int seeds64, int64_t n,
                                     void* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += stride) {
    int64_t d = 0;
    if (i < n) {
      const int64_t row = load_int(seeds, seeds64, i);
      d = load_int(indptr, indptr64, row + 1) - load_int(indptr, indptr64, row);
    }
    store_int(out, indptr64, i, d);
  }
}

// out[i] = indptr[seeds[i]]: where each selected row starts in the full edge array.
__global__ void subcsr_edge_base_kernel(const void* __restrict__ indptr, int indptr64,
                                        const void* __restrict__ seeds, int seeds64, int64_t n,
                                        void* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    store_int(out, indptr64, i, load_int(indptr, indptr64, load_int(seeds, seeds64, i)));
}

template <typename IxT>
__global__ void __launch_bounds__(256)
subcsr_fill_kernel(const void* __restrict__ indptr, int indptr64, const IxT* __restrict__ indices,
                   const void* __restrict__ seeds, int seeds64, int64_t n,
                   const void* __restrict__ gpu_indptr, IxT* __restrict__ out) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = threadIdx.x & 31;
  for (int64_t i = warp; i < n; i += n_warps) {
    const int64_t row = load_int(seeds, seeds64, i);
    const int64_t b = load_int(indptr, indptr64, row);
    const int64_t deg = load_int(indptr, indptr64, row + 1) - b;
    const IxT* src = indices + b;
    IxT* dst = out + load_int(gpu_indptr, indptr64, i);
    int64_t p = lane;
    for (; p + 96 < deg; p += 128) {  // four independent loads per lane in flight
      const IxT a0 = src[p], a1 = src[p + 32], a2 = src[p + 64], a3 = src[p + 96];
      dst[p] = a0;
      dst[p + 32] = a1;
      dst[p + 64] = a2;
      dst[p + 96] = a3;
    }
    for (; p < deg; p += 32) dst[p] = src[p];
  }
}

int launch_scan(shmt_ctx* ctx, void* data, int dtype, int64_t n, int exclusive,
                size_t scratch_off, cudaStream_t stream);
size_t scan_scratch_bytes(int64_t n);

// The fan-out a hop is laid out for: weighted picks take the lists of fan-outs up to 32, with
// replacement the warp-per-seed form of larger ones.
static int64_t hop_layout_k(bool weighted, bool replace, int64_t k) { return !weighted ? k : (replace ? 33 : 32); }

static int pick_seeds_per_tile(int64_t n, int64_t k) {
  int64_t s = (n + (int64_t)sm_count() * 4 - 1) / ((int64_t)sm_count() * 4);
  s = (s + kHopSeedStep - 1) / kHopSeedStep * kHopSeedStep;
  if (s < kHopSeedStep) s = kHopSeedStep;
  if (s > kMaxSeedsPerTile) s = kMaxSeedsPerTile;
  // with k <= 32 the list of a tile's neighbours takes at most 16 KB of shared memory
  const int64_t one_pass = k <= 8 ? 256 : (k <= 16 ? 128 : (k <= 32 ? 64 : kMaxSeedsPerTile));
  if (s > one_pass) s = one_pass;
  return (int)s;
}

// Fan-outs above 32 keep a set of chosen positions per warp in shared memory: the smallest
// power of two >= 2k words, for k <= 1024 (64 KB per CTA at most).  0: the fan-out needs none,
// or is too large for it.
constexpr int64_t kMaxSetPicks = 1024;
static uint32_t set_slots_for(int64_t k) {
  if (k <= 32 || k > kMaxSetPicks) return 0;
  uint32_t slots = 128;
  while ((int64_t)slots < 2 * k) slots <<= 1;
  return slots;
}

// The per-seed arrays of a tile and what lies behind them (see the kernel).
static size_t hop_smem_bytes(int seeds_per_tile, int64_t k, uint32_t set_slots, bool marks = false) {
  const size_t list = k <= 32 ? (size_t)seeds_per_tile * (size_t)k * sizeof(uint64_t) : 0;
  const size_t sets = (size_t)set_slots * sizeof(uint32_t) * (kHopThreads / 32);
  return (size_t)seeds_per_tile * (4 * sizeof(int64_t) + 1) + (list > sets ? list : sets) +
         (marks ? kMarkBuffer * sizeof(Mark) * (kHopThreads / 32) : 0);
}

template <typename IxT, int MODE>
static cudaError_t launch_hop_as(const HopJob& job, unsigned grid, size_t smem, cudaStream_t s, bool pdl) {
  if (!job.weights) {
    if (job.k <= 8) return launch_kernel(pdl, sample_hop_kernel<IxT, 8, MODE>, grid, kHopThreads, smem, s, job);
    if (job.k <= 16) return launch_kernel(pdl, sample_hop_kernel<IxT, 16, MODE>, grid, kHopThreads, smem, s, job);
  }
  if (smem > kPlainHopSmem) {
    static bool configured[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !configured[dev]) {
      const cudaError_t e =
          cudaFuncSetAttribute(sample_hop_kernel<IxT, 32, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)hop_smem_bytes(kMaxSeedsPerTile, 33, 2 * kMaxSetPicks));
      if (e != cudaSuccess) return e;
      configured[dev] = true;
    }
  }
  return launch_kernel(pdl, sample_hop_kernel<IxT, 32, MODE>, grid, kHopThreads, smem, s, job);
}

static bool on_device(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess) return a.type == cudaMemoryTypeDevice;
  cudaGetLastError();  // a failed query must not poison the next launch check
  return false;
}

template <typename IxT>
static cudaError_t launch_hop(HopJob job, int64_t n_tiles, cudaStream_t s, bool pdl = false) {
  const unsigned grid = (unsigned)n_tiles;
  job.set_slots = set_slots_for(job.k);
  const size_t smem = hop_smem_bytes(job.seeds_per_tile, hop_layout_k(job.weights, job.replace, job.k), job.set_slots,
                                     job.weights && !job.replace);
  if (job.rel_slots) return launch_hop_as<IxT, HOP_FUSED>(job, grid, smem, s, pdl);
  if (!job.weights && (job.n <= kTinyHostSeeds || (job.n <= kTinySeeds && on_device(job.indptr))))
    return launch_hop_as<IxT, HOP_TINY>(job, grid, smem, s, pdl);
  if (job.weights && !job.replace && job.post.host)  // the lists of fan-outs up to 32: within 48 KB
    return launch_kernel(pdl, sample_hop_kernel<IxT, 32, HOP_EARLY>, grid, kHopThreads, smem, s, job);
  return launch_hop_as<IxT, HOP_SINGLE>(job, grid, smem, s, pdl);
}

// Scratch layout of a multi-hop mini-batch, from its worst-case sizes (c_0 = n_seeds,
// c_{h+1} = c_h * (1 + fanouts[h])).
constexpr int kMaxHops = 8;
struct MinibatchPlan {
  int64_t cap[kMaxHops + 1], hop_tiles[kMaxHops], rel_tiles[kMaxHops];
  int spt[kMaxHops];
  size_t off_hop[kMaxHops], off_rel[kMaxHops];
  size_t scratch_bytes;
};

static int plan_minibatch(int64_t n_seeds, const int64_t* fanouts, int n_hops, MinibatchPlan* p,
                          bool weighted = false, bool replace = false) {
  SHMT_REQUIRE(n_hops >= 1 && n_hops <= kMaxHops, "mini-batch: 1..%d hops", kMaxHops);
  SHMT_REQUIRE(n_seeds >= 1 && n_seeds < ((int64_t)1 << 31), "mini-batch: seed count out of range");
  SHMT_REQUIRE(fanouts != nullptr, "mini-batch: fanouts is null");
  p->cap[0] = n_seeds;
  size_t cursor = ((size_t)(n_hops * 8 + 8) * 8 + 255) & ~(size_t)255;
  for (int h = 0; h < n_hops; ++h) {
    SHMT_REQUIRE(fanouts[h] >= 1 && fanouts[h] < ((int64_t)1 << 20), "mini-batch: fan-out out of range");
    p->cap[h + 1] = p->cap[h] * (1 + fanouts[h]);
    SHMT_REQUIRE(p->cap[h + 1] < ((int64_t)1 << 30), "mini-batch: worst-case frontier too large");
    p->spt[h] = pick_seeds_per_tile(p->cap[h], hop_layout_k(weighted, replace, fanouts[h]));
    p->hop_tiles[h] = (p->cap[h] + p->spt[h] - 1) / p->spt[h];
    p->rel_tiles[h] = (p->cap[h + 1] + kRelTile - 1) / kRelTile;
    p->off_hop[h] = cursor;
    cursor += (tile_state_bytes(p->hop_tiles[h]) + 255) & ~(size_t)255;
    p->off_rel[h] = cursor;
    cursor += (tile_state_bytes(p->rel_tiles[h]) + 255) & ~(size_t)255;
  }
  p->scratch_bytes = cursor;
  return SHMT_OK;
}

// Words for the ids of a mini-batch on a graph of `n_nodes` (0: not known): all or none.  None where a context
// that the caller has sized would have to grow.
static int64_t minibatch_words(const shmt_ctx* ctx, int64_t n_nodes) {
  if (n_nodes > kRelMaxWords) return 0;
  const bool fits = (size_t)n_nodes * sizeof(unsigned) <= ctx->words_bytes;
  return fits || !ctx->words_reserved ? n_nodes : 0;
}

}  // namespace shmt

using namespace shmt;

extern "C" {

int shmt_ctx_reserve_minibatch(shmt_ctx* ctx, int64_t n_seeds, const int64_t* fanouts, int n_hops,
                               void* stream) {
  return shmt_ctx_reserve_minibatch_nodes(ctx, n_seeds, fanouts, n_hops, 0, stream);
}

int shmt_ctx_reserve_minibatch_nodes(shmt_ctx* ctx, int64_t n_seeds, const int64_t* fanouts, int n_hops,
                                     int64_t n_nodes, void* stream) {
  SHMT_REQUIRE(ctx != nullptr, "shmt_ctx_reserve_minibatch: ctx is null");
  SHMT_REQUIRE(n_nodes >= 0, "shmt_ctx_reserve_minibatch: negative node count");
  // weighted hops without replacement have the smaller tiles, and so the more descriptors, of the two
  MinibatchPlan plan, weighted;
  if (int rc = plan_minibatch(n_seeds, fanouts, n_hops, &plan)) return rc;
  if (int rc = plan_minibatch(n_seeds, fanouts, n_hops, &weighted, /*weighted=*/true)) return rc;
  DeviceGuard guard(ctx->device);
  if (int rc = ctx_reserve(ctx, weighted.scratch_bytes > plan.scratch_bytes ? weighted.scratch_bytes : plan.scratch_bytes,
                           static_cast<cudaStream_t>(stream)))
    return rc;
  RelTable t;
  if (int rc = relabel_table(ctx, plan.cap[n_hops], &t, static_cast<cudaStream_t>(stream))) return rc;
  // and words, at least of as many nodes as fit in what a table takes beyond its slots: another graph may come
  const size_t slots = t.cap * sizeof(RelSlot), least = (size_t)4 << 20;
  size_t words = slots + slots / 2 < least ? least - slots : slots / 2;
  if (words > kRelMaxWords * sizeof(unsigned)) words = kRelMaxWords * sizeof(unsigned);
  if (n_nodes <= kRelMaxWords && words < n_nodes * sizeof(unsigned)) words = n_nodes * sizeof(unsigned);
  if (int rc = ctx_reserve_words(ctx, words, static_cast<cudaStream_t>(stream))) return rc;
  ctx->words_reserved = true;
  return SHMT_OK;
}

static int sample_hop_impl(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                           int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                           const shmt_map* map, const void* seeds, int seeds_dtype, int64_t n, int64_t k,
                           int replace, uint64_t rng_seed, uint64_t rng_offset, void* out_sub_indptr,
                           void* out_sub_indices, int64_t* nnz_host, void* stream, void* out_eids,
                           const void* gpu_edge_base, const float* weights = nullptr,
                           const float* gpu_weights = nullptr) {
  SHMT_REQUIRE(ctx != nullptr, "shmt_sample_hop: ctx is null");
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(indices_dtype) &&
                   valid_int_dtype(seeds_dtype),
               "shmt_sample_hop: ID can only be int32 or int64");
  SHMT_REQUIRE(n >= 0 && n < ((int64_t)1 << 31), "shmt_sample_hop: seed count out of range");
  SHMT_REQUIRE(k >= 0 && k < ((int64_t)1 << 31), "shmt_sample_hop: num_picks out of range");
  SHMT_REQUIRE(out_sub_indptr != nullptr, "shmt_sample_hop: out_sub_indptr is null");
  SHMT_REQUIRE(indptr != nullptr && (indices != nullptr || k == 0), "shmt_sample_hop: CSR is null");
  SHMT_REQUIRE(n == 0 || seeds != nullptr, "shmt_sample_hop: seeds are null");
  SHMT_REQUIRE(map == nullptr || (gpu_indptr != nullptr && gpu_indices != nullptr),
               "shmt_sample_hop: a map needs gpu_indptr and gpu_indices");
  SHMT_REQUIRE(n == 0 || k == 0 || out_sub_indices != nullptr,
               "shmt_sample_hop: out_sub_indices is null");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n == 0) {
    SHMT_CUDA_TRY(cudaMemsetAsync(out_sub_indptr, 0, int_itemsize(indptr_dtype), s));
    if (nnz_host) {
      SHMT_CUDA_TRY(cudaStreamSynchronize(s));
      *nnz_host = 0;
    }
    return SHMT_OK;
  }
  HopJob job{};
  job.indptr = indptr;
  job.indptr64 = indptr_dtype == SHMT_I64;
  job.indices = indices;
  job.gpu_indptr = gpu_indptr;
  job.gpu_indices = gpu_indices;
  job.map = view_of(map);
  job.seeds = seeds;
  job.seeds64 = seeds_dtype == SHMT_I64;
  job.n = n;
  job.k = k;
  job.replace = replace != 0;
  job.rng_seed = rng_seed;
  job.off_lo = (uint32_t)rng_offset;
  job.off_hi = (uint32_t)(rng_offset >> 32);
  job.sub_indptr = out_sub_indptr;
  job.sub_indices = out_sub_indices;
  job.out_eids = out_eids;
  job.gpu_edge_base = gpu_edge_base;
  job.weights = weights;
  job.gpu_weights = gpu_weights;
  job.seeds_per_tile = pick_seeds_per_tile(n, hop_layout_k(weights != nullptr, replace != 0, k));
  const int64_t n_tiles = (n + job.seeds_per_tile - 1) / job.seeds_per_tile;
  job.n_dev = nullptr;
  // Up to kSmallScanTiles tiles use look-back state that the kernel leaves at zero: no memset in front
  // (2 us and a gap on the GPU), and nothing behind the post that the scratch's next user waits for:
  // the state is zero again before the post, and what follows it writes the caller's outputs only.
  const bool small = n_tiles <= kSmallScanTiles;
  int64_t* done = nullptr;
  if (small) {
    job.ticket = ctx->scan_words();
    job.clean = done = ctx->scan_words() + 1;
    job.st = carve_tile_states(reinterpret_cast<char*>(ctx->scan_words() + 2), kSmallScanTiles);
  } else {
    if (int rc = ctx_reserve(ctx, tile_state_bytes(n_tiles), s)) return rc;
    done = ctx->d_words() + W_DONE;
    job.ticket = ctx->d_words() + W_TICKET;
    job.st = carve_tile_states(ctx->region(), n_tiles);
    SHMT_CUDA_TRY(cudaMemsetAsync(ctx->scratch, 0, 256 + tile_state_bytes(n_tiles), s));
  }
  job.status = ctx->d_words() + W_STATUS;
  job.result = ctx->d_words() + W_RESULT;
  if (nnz_host) job.post = ctx_begin_post(ctx, ctx->d_words(), 4, done);
  SHMT_CUDA_TRY(indices_dtype == SHMT_I64 ? launch_hop<long long>(job, n_tiles, s)
                                          : launch_hop<int>(job, n_tiles, s));
  SHMT_CUDA_TRY(cudaGetLastError());
  if (nnz_host) {
    if (!small) {
      if (int rc = ctx_mark_tail(ctx, s)) return rc;
    }
    if (int rc = ctx_await_post(ctx, job.post, s)) return rc;
    if (int rc = ctx_status_of_words(ctx, "shmt_sample_hop")) return rc;
    *nnz_host = ctx->h_words[W_RESULT];
  }
  return SHMT_OK;
}

int shmt_sample_hop(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                    int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                    const shmt_map* map, const void* seeds, int seeds_dtype, int64_t n, int64_t k,
                    int replace, uint64_t rng_seed, uint64_t rng_offset, void* out_sub_indptr,
                    void* out_sub_indices, int64_t* nnz_host, void* stream) {
  return sample_hop_impl(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map,
                         seeds, seeds_dtype, n, k, replace, rng_seed, rng_offset, out_sub_indptr,
                         out_sub_indices, nnz_host, stream, nullptr, nullptr);
}

int shmt_sample_hop_weighted(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                             int indices_dtype, const float* weights, const void* gpu_indptr,
                             const void* gpu_indices, const float* gpu_weights,
                             const void* gpu_edge_base, const shmt_map* map, const void* seeds,
                             int seeds_dtype, int64_t n, int64_t k, int replace, uint64_t rng_seed,
                             uint64_t rng_offset, void* out_sub_indptr, void* out_sub_indices,
                             void* out_edge_ids, int64_t* nnz_host, void* stream) {
  SHMT_REQUIRE(weights != nullptr || n == 0 || k == 0, "shmt_sample_hop_weighted: weights are null");
  SHMT_REQUIRE(replace || k <= 32,
               "shmt_sample_hop_weighted: without replacement the fan-out is limited to 32 (got %lld)",
               (long long)k);
  SHMT_REQUIRE(map == nullptr || gpu_weights != nullptr,
               "shmt_sample_hop_weighted: a cached graph needs gpu_weights");
  SHMT_REQUIRE(map == nullptr || out_edge_ids == nullptr || gpu_edge_base != nullptr,
               "shmt_sample_hop_weighted: edge ids of a cached graph need gpu_edge_base");
  return sample_hop_impl(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map,
                         seeds, seeds_dtype, n, k, replace, rng_seed, rng_offset, out_sub_indptr,
                         out_sub_indices, nnz_host, stream, out_edge_ids, gpu_edge_base, weights,
                         gpu_weights);
}

int shmt_sample_hop_eids(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                         int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                         const void* gpu_edge_base, const shmt_map* map, const void* seeds,
                         int seeds_dtype, int64_t n, int64_t k, int replace, uint64_t rng_seed,
                         uint64_t rng_offset, void* out_sub_indptr, void* out_sub_indices,
                         void* out_edge_ids, int64_t* nnz_host, void* stream) {
  SHMT_REQUIRE(n == 0 || k == 0 || out_edge_ids != nullptr, "shmt_sample_hop_eids: out_edge_ids is null");
  SHMT_REQUIRE(map == nullptr || gpu_edge_base != nullptr,
               "shmt_sample_hop_eids: a cached graph needs gpu_edge_base (shmt_subcsr_edge_base)");
  return sample_hop_impl(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map,
                         seeds, seeds_dtype, n, k, replace, rng_seed, rng_offset, out_sub_indptr,
                         out_sub_indices, nnz_host, stream, out_edge_ids, gpu_edge_base);
}

// Multi-hop mini-batch: every hop's sampling kernel and relabel kernels are queued back
// to back; each reads the size of its input from the device word the previous stage
// wrote, with grids sized for the largest frontier the fan-outs allow.  With `notes` the host hears of a
// hop's sizes as soon as its ids are counted, without them of all sizes at the end.
static int queue_minibatch(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                                 int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                                 const shmt_map* map, const void* seeds, int64_t n_seeds,
                                 const int64_t* fanouts, int n_hops, int replace, uint64_t rng_seed,
                                 uint64_t rng_offset, void* const* out_sub_indptr,
                                 void* const* out_sub_indices, void* const* out_relabel,
                                 void* const* out_frontier, void* stream,
                                 const void* gpu_edge_base, void* const* out_edge_ids,
                                 const float* weights = nullptr, const float* gpu_weights = nullptr,
                                 int64_t n_nodes = 0, bool notes = false) {
  SHMT_REQUIRE(ctx != nullptr, "shmt_sample_minibatch: ctx is null");
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(indices_dtype),
               "shmt_sample_minibatch: ID can only be int32 or int64");
  SHMT_REQUIRE(n_hops >= 1 && n_hops <= kMaxHops, "shmt_sample_minibatch: 1..%d hops", kMaxHops);
  SHMT_REQUIRE(n_seeds >= 1 && n_seeds < ((int64_t)1 << 31), "shmt_sample_minibatch: seed count out of range");
  SHMT_REQUIRE(indptr && indices && seeds && fanouts && out_sub_indptr && out_sub_indices &&
                   out_relabel && out_frontier,
               "shmt_sample_minibatch: null argument");
  SHMT_REQUIRE(map == nullptr || (gpu_indptr != nullptr && gpu_indices != nullptr),
               "shmt_sample_minibatch: a map needs gpu_indptr and gpu_indices");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);

  // worst-case frontier sizes and the scratch plan: [words][per hop: sample tiles | relabel tiles]
  MinibatchPlan plan;
  if (int rc = plan_minibatch(n_seeds, fanouts, n_hops, &plan, weights != nullptr, replace != 0)) return rc;
  for (int h = 0; h < n_hops; ++h)
    SHMT_REQUIRE(out_sub_indptr[h] && out_sub_indices[h] && out_relabel[h] && out_frontier[h],
                 "shmt_sample_minibatch: output buffer of hop %d is null", h);
  const int64_t* cap = plan.cap;
  const int64_t *hop_tiles = plan.hop_tiles, *rel_tiles = plan.rel_tiles;
  const int* spt = plan.spt;
  const size_t *off_hop = plan.off_hop, *off_rel = plan.off_rel;
  const size_t cursor = plan.scratch_bytes;
  // Every batch has tags of its own, which a replay would use again; and nobody can wait for the sizes.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  SHMT_CUDA_TRY(cudaStreamIsCapturing(s, &capture));
  SHMT_REQUIRE(capture == cudaStreamCaptureStatusNone, "shmt_sample_minibatch: the stream is being captured");
  if (int rc = ctx_reserve(ctx, cursor, s)) return rc;
  char* base = ctx->region();
  int64_t* words = reinterpret_cast<int64_t*>(base);
  SHMT_CUDA_TRY(cudaMemsetAsync(base, 0, cursor, s));  // words, tickets and every tile descriptor
  int64_t* status = words + n_hops * 8;

  // the relabel table for the largest hop, reserved before anything is queued
  RelWords rel_words;
  rel_words.n = minibatch_words(ctx, n_nodes);
  {
    RelTable biggest;
    if (int rc = relabel_table(ctx, cap[n_hops], &biggest, s)) return rc;
  }
  if (rel_words.n) {
    if (int rc = ctx_reserve_words(ctx, (size_t)rel_words.n * sizeof(unsigned), s)) return rc;
    unsigned ids = 0;
    for (int h = 0; h < n_hops; ++h) ids += (unsigned)cap[h + 1];
    if (int rc = ctx_take_tags(ctx, ids, &rel_words.tag, s)) return rc;
    rel_words.tag += ids;  // goes down hop by hop
  }
  const void* cur_seeds = seeds;
  HostPost post{};
  RelRepeats repeats{};
  repeats.words = words;
  repeats.n_seeds = n_seeds;
  ctx->batch.n_hops = 0;
  ctx->batch.noted = notes;
  for (int h = 0; h < n_hops; ++h) {
    int64_t* w = words + h * 8;  // [0] hop ticket, [1] nnz, [2] relabel ticket, [3] n_unique, [4] CTAs done
    HopJob job{};
    job.indptr = indptr;
    job.indptr64 = indptr_dtype == SHMT_I64;
    job.indices = indices;
    job.gpu_indptr = gpu_indptr;
    job.gpu_indices = gpu_indices;
    job.map = view_of(map);
    job.seeds = cur_seeds;
    job.seeds64 = indices_dtype == SHMT_I64;
    job.n = h == 0 ? n_seeds : 0;
    job.n_dev = h == 0 ? nullptr : words + (h - 1) * 8 + 3;
    job.k = fanouts[h];
    job.replace = replace != 0;
    job.rng_seed = rng_seed;
    job.off_lo = (uint32_t)(rng_offset + h);
    job.off_hi = (uint32_t)((rng_offset + h) >> 32);
    job.sub_indptr = out_sub_indptr[h];
    job.sub_indices = out_sub_indices[h];
    job.seeds_per_tile = spt[h];
    job.out_eids = out_edge_ids ? out_edge_ids[h] : nullptr;
    job.gpu_edge_base = gpu_edge_base;
    job.weights = weights;
    job.gpu_weights = gpu_weights;
    job.st = carve_tile_states(base + off_hop[h], hop_tiles[h]);
    job.ticket = w + 0;
    job.status = status;
    job.result = w + 1;
    RelTable t;  // every sampler claims the relabel slots of what it emits
    if (rel_words.n) rel_words.tag -= (unsigned)cap[h + 1];
    if (int rc = relabel_table(ctx, cap[h + 1], &t, s, rel_words)) return rc;
    job.rel_slots = t.slots;
    job.rel_cap = t.cap;
    job.rel_words = t.words;
    job.rel_n_words = t.n_words;
    job.rel_tag = t.tag;
    job.rel_out = out_relabel[h];
    SHMT_CUDA_TRY(indices_dtype == SHMT_I64 ? launch_hop<long long>(job, hop_tiles[h], s, /*pdl=*/h > 0)
                                            : launch_hop<int>(job, hop_tiles[h], s, /*pdl=*/h > 0));
    SHMT_CUDA_TRY(cudaGetLastError());

    Parts ps{};
    ps.n = 2;
    ps.is64 = indices_dtype == SHMT_I64;
    ps.ptr[0] = cur_seeds;
    ps.ptr[1] = out_sub_indices[h];
    ps.start[1] = n_seeds;  // used for hop 0 only, whose seed count the host knows
    ps.dev_n0 = h == 0 ? nullptr : words + (h - 1) * 8 + 3;
    ps.dev_n1 = w + 1;
    // every size and the status word are final once the last hop's ids are counted: that kernel hands them
    // to the host, which returns while the numbers of the repeats are still being written
    if (h == n_hops - 1)
      post = ctx_begin_post(ctx, words, n_hops * 8 + 8, w + 4);
    else
      post = notes ? ctx_begin_note(ctx, kNoteWord + 2 * h) : HostPost{};
    if (h < n_hops - 1 && !post.host) ctx->batch.noted = false;
    if (int rc = launch_relabel(ctx, ps, cap[h + 1], out_frontier[h], out_relabel[h],
                                carve_tile_states(base + off_rel[h], rel_tiles[h]), w + 2, status,
                                w + 3, s, /*inserted=*/true, /*pdl=*/true, &post, /*survey=*/nullptr, rel_words))
      return rc;
    repeats.out[h] = out_relabel[h];
    cur_seeds = out_frontier[h];
  }
  if (rel_words.n) {
    repeats.n_hops = n_hops;
    if (int rc = launch_relabel_repeats(repeats, cap + 1, indices_dtype == SHMT_I64, s)) return rc;
  }
  if (int rc = ctx_mark_tail(ctx, s)) return rc;
  ctx->batch.post = post;
  ctx->batch.stream = stream;
  ctx->batch.n_hops = n_hops;
  ctx->batch.n_seeds = n_seeds;
  return SHMT_OK;
}

// Waits for the end of the queued mini-batch: all sizes are in ctx->h_words then.
static int await_minibatch(shmt_ctx* ctx) {
  const int n_hops = ctx->batch.n_hops;
  SHMT_REQUIRE(n_hops > 0, "mini-batch: none has been started");
  ctx->batch.n_hops = 0;
  if (int rc = ctx_await_post(ctx, ctx->batch.post, static_cast<cudaStream_t>(ctx->batch.stream))) return rc;
  const int64_t st = ctx->h_words[n_hops * 8];
  if (st != DEV_OK) {
    ctx_table_failed(ctx);
    set_error("shmt_sample_minibatch: device status %lld (%s)", (long long)st,
              st == DEV_TIMEOUT ? "a bounded look-back wait ran out" : "relabel table overflow");
    return st == DEV_TIMEOUT ? SHMT_ERR_TIMEOUT : SHMT_ERR_CAPACITY;
  }
  return SHMT_OK;
}

// {seeds in, edges sampled, distinct ids out} of hop `h`, from the words of a mini-batch that is over.
static void hop_sizes(const shmt_ctx* ctx, int h, int64_t* sizes) {
  sizes[0] = h == 0 ? ctx->batch.n_seeds : ctx->h_words[(h - 1) * 8 + 3];
  sizes[1] = ctx->h_words[h * 8 + 1];
  sizes[2] = ctx->h_words[h * 8 + 3];
}

static int finish_minibatch(shmt_ctx* ctx, int64_t* sizes_host) {
  const int n_hops = ctx->batch.n_hops;
  if (int rc = await_minibatch(ctx)) return rc;
  for (int h = 0; h < n_hops; ++h) hop_sizes(ctx, h, sizes_host + 3 * h);
  return SHMT_OK;
}

int shmt_sample_minibatch(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                          int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                          const shmt_map* map, const void* seeds, int64_t n_seeds,
                          const int64_t* fanouts, int n_hops, int replace, uint64_t rng_seed,
                          uint64_t rng_offset, void* const* out_sub_indptr,
                          void* const* out_sub_indices, void* const* out_relabel,
                          void* const* out_frontier, int64_t* sizes_host, void* stream) {
  SHMT_REQUIRE(sizes_host != nullptr, "shmt_sample_minibatch: null argument");
  if (int rc = queue_minibatch(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map, seeds,
                               n_seeds, fanouts, n_hops, replace, rng_seed, rng_offset, out_sub_indptr,
                               out_sub_indices, out_relabel, out_frontier, stream, nullptr, nullptr))
    return rc;
  return finish_minibatch(ctx, sizes_host);
}

int shmt_sample_minibatch_eids(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                               int indices_dtype, const void* gpu_indptr, const void* gpu_indices,
                               const void* gpu_edge_base, const shmt_map* map, const void* seeds,
                               int64_t n_seeds, const int64_t* fanouts, int n_hops, int replace,
                               uint64_t rng_seed, uint64_t rng_offset, void* const* out_sub_indptr,
                               void* const* out_sub_indices, void* const* out_edge_ids,
                               void* const* out_relabel, void* const* out_frontier,
                               int64_t* sizes_host, void* stream) {
  SHMT_REQUIRE(out_edge_ids != nullptr, "shmt_sample_minibatch_eids: out_edge_ids is null");
  SHMT_REQUIRE(map == nullptr || gpu_edge_base != nullptr,
               "shmt_sample_minibatch_eids: a cached graph needs gpu_edge_base (shmt_subcsr_edge_base)");
  for (int h = 0; h < n_hops && h < 8; ++h)
    SHMT_REQUIRE(out_edge_ids[h] != nullptr, "shmt_sample_minibatch_eids: edge-id buffer of hop %d is null", h);
  SHMT_REQUIRE(sizes_host != nullptr, "shmt_sample_minibatch_eids: null argument");
  if (int rc = queue_minibatch(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map, seeds,
                               n_seeds, fanouts, n_hops, replace, rng_seed, rng_offset, out_sub_indptr,
                               out_sub_indices, out_relabel, out_frontier, stream, gpu_edge_base, out_edge_ids))
    return rc;
  return finish_minibatch(ctx, sizes_host);
}

int shmt_sample_minibatch_weighted(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* indices,
                                   int indices_dtype, const float* weights, const void* gpu_indptr,
                                   const void* gpu_indices, const float* gpu_weights, const shmt_map* map,
                                   const void* seeds, int64_t n_seeds, const int64_t* fanouts, int n_hops,
                                   int replace, uint64_t rng_seed, uint64_t rng_offset,
                                   void* const* out_sub_indptr, void* const* out_sub_indices,
                                   void* const* out_relabel, void* const* out_frontier, int64_t* sizes_host,
                                   void* stream) {
  SHMT_REQUIRE(weights != nullptr, "shmt_sample_minibatch_weighted: weights are null");
  SHMT_REQUIRE(map == nullptr || gpu_weights != nullptr,
               "shmt_sample_minibatch_weighted: a cached graph needs gpu_weights");
  for (int h = 0; fanouts && h < n_hops && h < 8; ++h)
    SHMT_REQUIRE(replace || fanouts[h] <= 32,
                 "shmt_sample_minibatch_weighted: without replacement the fan-out is at most 32 (hop %d has %lld)", h,
                 (long long)fanouts[h]);
  SHMT_REQUIRE(sizes_host != nullptr, "shmt_sample_minibatch_weighted: null argument");
  if (int rc = queue_minibatch(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map, seeds,
                               n_seeds, fanouts, n_hops, replace, rng_seed, rng_offset, out_sub_indptr,
                               out_sub_indices, out_relabel, out_frontier, stream, nullptr, nullptr, weights,
                               gpu_weights))
    return rc;
  return finish_minibatch(ctx, sizes_host);
}

int shmt_minibatch_start(shmt_ctx* ctx, const void* indptr, int indptr_dtype, int64_t n_nodes, const void* indices,
                         int indices_dtype, const float* weights, const void* gpu_indptr, const void* gpu_indices,
                         const float* gpu_weights, const void* gpu_edge_base, const shmt_map* map, const void* seeds,
                         int64_t n_seeds, const int64_t* fanouts, int n_hops, int replace, uint64_t rng_seed,
                         uint64_t rng_offset, void* indptr_pool, void* indices_pool, const int64_t* layout,
                         int with_edge_ids, void* stream) {
  SHMT_REQUIRE(n_hops >= 1 && n_hops <= kMaxHops, "shmt_minibatch_start: 1..%d hops", kMaxHops);
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(indices_dtype),
               "shmt_minibatch_start: ID can only be int32 or int64");
  SHMT_REQUIRE(indptr_pool && indices_pool && layout, "shmt_minibatch_start: null argument");
  SHMT_REQUIRE(n_nodes >= 0, "shmt_minibatch_start: negative node count");
  SHMT_REQUIRE(!weights || !with_edge_ids, "shmt_minibatch_start: weights and edge ids cannot be combined");
  SHMT_REQUIRE(!with_edge_ids || map == nullptr || gpu_edge_base != nullptr,
               "shmt_minibatch_start: edge ids of a cached graph need gpu_edge_base (shmt_subcsr_edge_base)");
  SHMT_REQUIRE(!weights || map == nullptr || gpu_weights != nullptr,
               "shmt_minibatch_start: a cached graph needs gpu_weights");
  for (int h = 0; weights && fanouts && h < n_hops; ++h)
    SHMT_REQUIRE(replace || fanouts[h] <= 32,
                 "shmt_minibatch_start: without replacement the fan-out is at most 32 (hop %d has %lld)", h,
                 (long long)fanouts[h]);
  void *sub_indptr[kMaxHops], *sub_indices[kMaxHops], *relabel[kMaxHops], *frontier[kMaxHops], *edge_ids[kMaxHops];
  char *p = static_cast<char*>(indptr_pool), *x = static_cast<char*>(indices_pool);
  const int p_item = int_itemsize(indptr_dtype), x_item = int_itemsize(indices_dtype);
  for (int h = 0; h < n_hops; ++h) {
    sub_indptr[h] = p + layout[h] * p_item;
    edge_ids[h] = with_edge_ids ? p + layout[n_hops + h] * p_item : nullptr;
    sub_indices[h] = x + layout[2 * n_hops + h] * x_item;
    relabel[h] = x + layout[3 * n_hops + h] * x_item;
    frontier[h] = x + layout[4 * n_hops + h] * x_item;
  }
  return queue_minibatch(ctx, indptr, indptr_dtype, indices, indices_dtype, gpu_indptr, gpu_indices, map, seeds, n_seeds,
                         fanouts, n_hops, replace, rng_seed, rng_offset, sub_indptr, sub_indices, relabel, frontier,
                         stream, gpu_edge_base, with_edge_ids ? edge_ids : nullptr, weights, gpu_weights, n_nodes,
                         /*notes=*/true);
}

int shmt_minibatch_hop(shmt_ctx* ctx, int hop, int64_t* sizes_host) {
  SHMT_REQUIRE(ctx != nullptr && sizes_host != nullptr, "shmt_minibatch_hop: null argument");
  const int n_hops = ctx->batch.n_hops;
  SHMT_REQUIRE(n_hops > 0 && hop >= 0 && hop < n_hops, "shmt_minibatch_hop: no such hop has been started");
  DeviceGuard guard(ctx->device);
  if (hop < n_hops - 1 && ctx->batch.noted) {
    int rc = SHMT_OK;
    for (int h = hop > 0 ? hop - 1 : 0; h <= hop && rc == SHMT_OK; ++h)
      rc = ctx_await_note(ctx, kNoteWord + 2 * h, static_cast<cudaStream_t>(ctx->batch.stream));
    if (rc > 0) return rc;
    if (rc == SHMT_OK) {
      sizes_host[0] = hop == 0 ? ctx->batch.n_seeds : ctx->h_words[kNoteWord + 2 * hop - 1];
      sizes_host[1] = ctx->h_words[kNoteWord + 2 * hop];
      sizes_host[2] = ctx->h_words[kNoteWord + 2 * hop + 1];
      return SHMT_OK;
    }
  }
  if (int rc = await_minibatch(ctx)) return rc;
  if (hop < n_hops - 1) ctx->batch.n_hops = n_hops;  // the others may be asked for
  hop_sizes(ctx, hop, sizes_host);
  return SHMT_OK;
}

int shmt_subcsr_count(shmt_ctx* ctx, const void* indptr, int indptr_dtype, const void* seeds,
                      int seeds_dtype, int64_t n, void* out_gpu_indptr, int64_t* nnz_host,
                      void* stream) {
  SHMT_REQUIRE(ctx != nullptr, "shmt_subcsr_count: ctx is null");
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(seeds_dtype),
               "shmt_subcsr_count: ID can only be int32 or int64");
  SHMT_REQUIRE(n >= 0, "shmt_subcsr_count: negative count");
  SHMT_REQUIRE(indptr && out_gpu_indptr && (n == 0 || seeds), "shmt_subcsr_count: null argument");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (int rc = ctx_reserve(ctx, scan_scratch_bytes(n + 1), s)) return rc;
  int64_t blocks = (n + 1 + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  subcsr_degree_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(
      indptr, indptr_dtype == SHMT_I64, seeds, seeds_dtype == SHMT_I64, n, out_gpu_indptr);
  SHMT_CUDA_TRY(cudaGetLastError());
  if (int rc = launch_scan(ctx, out_gpu_indptr, indptr_dtype, n + 1, /*exclusive=*/1, 0, s))
    return rc;
  if (nnz_host) {
    int64_t last = 0;
    const int sz = int_itemsize(indptr_dtype);
    SHMT_CUDA_TRY(cudaMemcpyAsync(&last, static_cast<char*>(out_gpu_indptr) + (size_t)n * sz, sz,
                                  cudaMemcpyDeviceToHost, s));
    if (int rc = ctx_fetch_words(ctx, s, "shmt_subcsr_count")) return rc;
    *nnz_host = indptr_dtype == SHMT_I64 ? last : (int64_t)(int32_t)last;
  }
  return SHMT_OK;
}

int shmt_subcsr_edge_base(const void* indptr, int indptr_dtype, const void* seeds, int seeds_dtype,
                          int64_t n, void* out_edge_base, void* stream) {
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(seeds_dtype),
               "shmt_subcsr_edge_base: ID can only be int32 or int64");
  SHMT_REQUIRE(n >= 0, "shmt_subcsr_edge_base: negative count");
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(indptr && seeds && out_edge_base, "shmt_subcsr_edge_base: null argument");
  int64_t blocks = (n + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 16;
  subcsr_edge_base_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      indptr, indptr_dtype == SHMT_I64, seeds, seeds_dtype == SHMT_I64, n, out_edge_base);
  SHMT_CUDA_TRY(cudaGetLastError());
  return SHMT_OK;
}

int shmt_subcsr_fill(const void* indptr, int indptr_dtype, const void* indices, int indices_dtype,
                     const void* seeds, int seeds_dtype, int64_t n, const void* gpu_indptr,
                     void* out_gpu_indices, void* stream) {
  SHMT_REQUIRE(valid_int_dtype(indptr_dtype) && valid_int_dtype(indices_dtype) &&
                   valid_int_dtype(seeds_dtype),
               "shmt_subcsr_fill: ID can only be int32 or int64");
  SHMT_REQUIRE(n >= 0, "shmt_subcsr_fill: negative count");
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(indptr && indices && seeds && gpu_indptr, "shmt_subcsr_fill: null argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t blocks = (n + 7) / 8;
  const int64_t cap = (int64_t)sm_count() * 32;
  const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
  if (indices_dtype == SHMT_I64)
    subcsr_fill_kernel<long long><<<grid, 256, 0, s>>>(
        indptr, indptr_dtype == SHMT_I64, static_cast<const long long*>(indices), seeds,
        seeds_dtype == SHMT_I64, n, gpu_indptr, static_cast<long long*>(out_gpu_indices));
  else
    subcsr_fill_kernel<int><<<grid, 256, 0, s>>>(
        indptr, indptr_dtype == SHMT_I64, static_cast<const int*>(indices), seeds,
        seeds_dtype == SHMT_I64, n, gpu_indptr, static_cast<int*>(out_gpu_indices));
  SHMT_CUDA_TRY(cudaGetLastError());
  return SHMT_OK;
}

}  // extern "C"
