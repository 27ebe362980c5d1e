// Unique (first-occurrence order) + dense remap of concatenated id arrays.
// Same result as the reference's TensorRelabel (src/tensor_relabel.cu:125-209):
// unique[j] is the j-th distinct id in order of first appearance and
// relabel[i] is the position of input[i] in unique.
//
// Three kernels instead of the reference's cat + 2 fills + 4 thrust passes + CUB
// scan: (1) claim a table slot per distinct id and take the minimum input
// index per slot, remembering each element's slot in the output array;
// (2) flag first occurrences, scan the flags with a decoupled look-back inside
// the same kernel, emit unique ids and the slot -> new id table, and put every slot
// that was used back to "empty", so the table needs no memset between calls;
// (3) remap the repeats.  Every element probes the table once (the reference four times).
// Up to 4,096 ids are one CTA's work; more than 2^20 are looked over first and use the smallest
// form of the table their ids allow, (2) becomes three kernels without a look-back, and a last one
// empties what (3) leaves of the small forms.
// The element counts may live on the device (written by an earlier kernel), so a
// chain of hops can be queued without the host knowing any size.
#include <type_traits>

#include "relabel.cuh"

namespace shmt {

constexpr uint64_t kRelSurveyMinTableBytes = 32ull << 20;

// Sizes of the input: the host's, or in the two-part form those an earlier kernel left on the device.
// Kept beside the parts, which stay the launch's constants: written back into them they would live
// in local memory, and so would every access by part number (a compact kernel over 300,000 ids spent
// most of its 32 us queueing for that; see part_elem).
struct PartSizes {
  int64_t numel;
  int64_t split;  // two-part form: elements of part 0; else -1
};
__device__ __forceinline__ PartSizes resolve_sizes(const Parts& ps) {
  if (!ps.dev_n1) return PartSizes{ps.start[kMaxParts], -1};
  const int64_t a = ps.dev_n0 ? *ps.dev_n0 : ps.start[1];
  return PartSizes{a + *ps.dev_n1, a};
}

__device__ __forceinline__ int64_t part_elem(const Parts& ps, const PartSizes& sz, int64_t i) {
  const void* p = ps.ptr[0];
  int64_t from = 0;
  if (sz.split >= 0) {
    if (i >= sz.split) {
      p = ps.ptr[1];
      from = sz.split;
    }
  } else if (ps.n > 1) {
#pragma unroll
    for (int q = 1; q < kMaxParts; ++q)
      if (q < ps.n && i >= ps.start[q]) {
        p = ps.ptr[q];
        from = ps.start[q];
      }
  }
  return load_int(p, ps.is64, i - from);
}

// One id in 2^shift is in the sample, picked by its hash, so that all its occurrences are or none
// is; at most 2^(kRelSampleBits - 1) of the ids then are, and the bitmap stays sparse enough to
// count them by the bits they set (linear counting, Whang et al. 1990).
__device__ __forceinline__ int relabel_sample_shift(int64_t numel) {
  int shift = 0;
  while ((numel >> shift) > ((int64_t)1 << (kRelSampleBits - 1))) ++shift;
  return shift;
}

// A look at a large input before any slot is claimed: its largest id (a negative id counts as
// huge), and how many distinct ids it holds, from a sample.  A sampled id that many elements share would be
// looked up in the bitmap, one sector of L2, by every warp (3,000,000 ids, a tenth of them the same: 38 us
// for 24 without such ids); a CTA therefore remembers what it has looked up.
constexpr int kRelKnown = 1024;
__global__ void __launch_bounds__(kRelThreads, 8)
relabel_survey_kernel(Parts ps, RelSurvey* survey, LaunchPad<56>) {
  __shared__ unsigned s_marked[kRelThreads / 32];
  __shared__ unsigned long long s_largest[kRelThreads / 32];
  __shared__ uint32_t s_known[kRelKnown];  // bits this CTA has looked up or set, the last at each place
  pdl_prologue();
  for (int q = (int)threadIdx.x; q < kRelKnown; q += kRelThreads) s_known[q] = ~0u;
  __syncthreads();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  const int shift = relabel_sample_shift(numel);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long m = 0;
  unsigned marked = 0;
  auto take = [&](long long id) {
    m = max(m, (unsigned long long)id);
    const uint64_t h = mix64((uint64_t)id);
    if (shift == 0 || (h >> (64 - shift)) == 0) {
      const uint32_t at = (uint32_t)h & ((1u << kRelSampleBits) - 1u), bit = 1u << (at & 31);
      volatile uint32_t* known = s_known + at % kRelKnown;
      if (*known == at) return;
      *known = at;
      if (!(__ldcg(survey->bitmap + (at >> 5)) & bit) && relabel_lowest(at))
        marked += (atomicOr(survey->bitmap + (at >> 5), bit) & bit) == 0;
    }
  };
#pragma unroll
  for (int p = 0; p < kMaxParts; ++p) {
    if (p >= ps.n) break;
    const int64_t n = ps.start[p + 1] - ps.start[p];
    int64_t done = 0;  // elements covered by the 16-byte loads below
    if ((reinterpret_cast<uintptr_t>(ps.ptr[p]) & 15) == 0) {
      // an aligned part: 16-byte loads, two per thread in flight (four at 5 CTAs per SM: 77 us for 71)
      constexpr int U = 2;
      const int per = ps.is64 ? 2 : 4;
      const int64_t n_vec = n / per;
      const uint4* src = static_cast<const uint4*>(ps.ptr[p]);
      for (int64_t v = gtid; v < n_vec; v += U * stride) {
        uint4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v + u * stride < n_vec) x[u] = __ldg(src + v + u * stride);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (v + u * stride >= n_vec) continue;
          if (ps.is64) {
            take((long long)(((unsigned long long)x[u].y << 32) | x[u].x));
            take((long long)(((unsigned long long)x[u].w << 32) | x[u].z));
          } else {
            take((int)x[u].x);
            take((int)x[u].y);
            take((int)x[u].z);
            take((int)x[u].w);
          }
        }
      }
      done = n_vec * per;
    }
    for (int64_t i = done + gtid; i < n; i += stride) take(load_int(ps.ptr[p], ps.is64, i));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    marked += __shfl_xor_sync(0xffffffffu, marked, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_marked[threadIdx.x >> 5] = marked;
    s_largest[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    marked = 0;
    for (int w = 0; w < kRelThreads / 32; ++w) {
      marked += s_marked[w];
      m = max(m, s_largest[w]);
    }
    if (m > __ldcg(&survey->largest)) atomicMax(&survey->largest, m);
    if (marked) atomicAdd(&survey->marked, (unsigned long long)marked);
  }
}

// How a call of `numel` ids uses the table.  Without a survey: at least two slots per id, as if all
// were distinct.  With one: kRelSlotsPerId slots per distinct id; or, where fewer bytes per id do:
// * ids that are all smaller than the table are places themselves (densely numbered nodes): one word
//   per id, its smallest index, is all there is to keep (RelSmall::stride 1);
// * ids of few enough bits are kept in half-size slots where full ones would outgrow the L2 cache
//   (RelSmall::stride 2).
constexpr double kRelSlotsPerId = 2.0;

// Half-size slots.  An id of b bits is mapped one to one onto another number of b bits, whose top bits
// are the home quad (four slots, 32 bytes) and whose other bits, with the distance from home, are all
// the slot has to hold to tell the id: {tag 32, first 32} instead of {id 64, first 32, new id 32}.  The
// new id takes the place of `first`, marked so that no index equals it.  What bounds a large relabel is
// the sectors its random accesses draw from HBM (2.9 TB/s of them is all there is); half the table
// means fewer.  An id that finds its 31 quads full goes to an ordinary slot behind them.
struct RelSmall {
  unsigned* words;  // the front of the table; nullptr: ordinary slots are used
  uint32_t n;       // places
  int stride;       // words per place: 1 = the id is the place, 2 = half-size slot
  int bits, quad_bits;
  RelRange rest;    // ordinary slots behind half-size ones; a position is n + index there
};
constexpr int kHalfRemainderBits = 26, kHalfQuads = 31;  // the tag is never all ones, which is an empty slot's
constexpr double kHalfSlotsPerId = 1.6;                  // before rounding up to a power of two
constexpr double kHalfMinBytes = 40.0 * (1 << 20);       // ordinary slots of this much are in L2 anyway

struct RelUse {
  RelRange range;
  RelSmall small;
};
__device__ __forceinline__ RelUse relabel_use(const RelTable& t, int64_t numel, const RelSurvey* survey) {
  RelUse u;
  u.small = RelSmall{nullptr, 0, 0, 0, 0, {}};
  u.range = RelRange{t.slots, relabel_near((double)numel, relabel_slots_per_id((double)numel, 2.0), t.cap), t.cap};
  if (!survey) return u;
  if (survey->largest < (unsigned long long)t.cap) {
    u.small = RelSmall{reinterpret_cast<unsigned*>(t.slots), (uint32_t)survey->largest + 1, 1, 0, 0, {}};
    return u;
  }
  const float bits = (float)(1 << kRelSampleBits), free_bits = bits - (float)survey->marked;
  const float sampled = free_bits > 0.0f ? -bits * logf(free_bits / bits) : bits * 16.0f;
  double ids = (double)sampled * (double)(1ull << relabel_sample_shift(numel));
  if (ids > (double)numel) ids = (double)numel;
  u.range.near = relabel_near(ids, kRelSlotsPerId, t.cap);
  if (ids * kRelSlotsPerId * sizeof(RelSlot) < kHalfMinBytes || t.cap > (1u << 30)) return u;
  int quad_bits = 0;
  while ((double)(4ull << quad_bits) < ids * kHalfSlotsPerId) ++quad_bits;
  int id_bits = 64 - __clzll((long long)survey->largest);
  if (id_bits < quad_bits) id_bits = quad_bits;
  if (id_bits - quad_bits > kHalfRemainderBits) return u;
  // The ordinary slots behind the n places would hold every id of the call, whatever the survey saw and wherever
  // the homes lie: cap / 2 is a power of two P >= numel, and n / 2, a power of two below 1.6 * numel, is
  // at most P, so that cap - n / 2 >= numel.
  const uint32_t n = 4u << quad_bits, rest = t.cap - n / 2;
  u.small = RelSmall{reinterpret_cast<unsigned*>(t.slots), n, 2, id_bits, quad_bits,
                     RelRange{t.slots + n / 2, rest, rest}};
  return u;
}

// One to one on numbers of `bits` bits: every step can be undone (a right shift by half of the bits,
// a product with an odd number modulo 2^bits).
__device__ __forceinline__ uint64_t mix_bits(uint64_t x, int bits) {
  const uint64_t mask = bits >= 64 ? ~0ull : (1ull << bits) - 1;
  const int half = (bits + 1) / 2;
  x ^= x >> half;
  x = (x * 0xff51afd7ed558ccdULL) & mask;
  x ^= x >> half;
  x = (x * 0xc4ceb9fe1a85ec53ULL) & mask;
  x ^= x >> half;
  return x;
}

// relabel_enter for half-size slots: a claim enters the index with the id.
__device__ __forceinline__ uint32_t relabel_claim_half(const RelSmall& t, long long key, unsigned i, int64_t* status,
                                                       bool* maybe_first) {
  const uint64_t x = mix_bits((uint64_t)key, t.bits);
  const int low = t.bits - t.quad_bits;
  const uint32_t home = (uint32_t)(x >> low), remainder = (uint32_t)(x & ((1ull << low) - 1));
  const uint32_t quads = t.n / 4;
  unsigned long long* slots = reinterpret_cast<unsigned long long*>(t.words);
  for (uint32_t d = 0; d < kHalfQuads; ++d) {
    const uint32_t at = ((home + d) & (quads - 1)) * 4, tag = (d << kHalfRemainderBits) | remainder;
    unsigned long long w[4];
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3])
                 : "l"(slots + at)
                 : "memory");
    int found = -1;
    unsigned seen = 0xFFFFFFFFu;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (found >= 0) continue;
      if ((uint32_t)(w[q] >> 32) == ~0u) {  // empty, whatever an ordinary slot has left below
        const unsigned long long empty = w[q];
        w[q] = atomicCAS(slots + at + q, empty, ((unsigned long long)tag << 32) | i);
        if (w[q] == empty) {
          *maybe_first = true;
          return at + q;
        }
      }
      if ((uint32_t)(w[q] >> 32) == tag) {
        found = q;
        seen = (unsigned)w[q];
      }
    }
    if (found >= 0) {
      *maybe_first = seen > i;
      if (seen > i) atomicMin(t.words + 2 * (size_t)(at + found), i);
      return at + found;
    }
  }
  return t.n + relabel_enter<true>(t.rest, key, i, status, maybe_first);
}

// Where the later passes of a surveyed call find what they need at position `pos`.
struct RelView {
  RelSmall small;
  RelSlot* slots;  // ordinary slots, by position
  __device__ __forceinline__ RelView(const RelTable& t, int64_t numel, const RelSurvey* survey) {
    small = relabel_use(t, numel, survey).small;
    slots = small.words ? small.rest.slots - small.n : t.slots;  // only indexed from small.n on
  }
  __device__ __forceinline__ unsigned* word(uint32_t pos) const { return small.words + (size_t)pos * small.stride; }
  __device__ __forceinline__ unsigned first(uint32_t pos) const {
    return __ldcg(pos < small.n ? word(pos) : &slots[pos].first);
  }
  __device__ __forceinline__ unsigned newid(uint32_t pos) const { return first(pos) & ~kRelNewId; }
  __device__ __forceinline__ void number(uint32_t pos, unsigned uid) const {
    if (pos < small.n)
      *word(pos) = uid | kRelNewId;
    else
      *reinterpret_cast<uint4*>(slots + pos) = make_uint4(~0u, ~0u, uid | kRelNewId, ~0u);
  }
};

constexpr uint32_t kNoSlot = 0xFFFFFFFFu;
constexpr unsigned kRelSms = 148, kRelInsertCtas = 7;  // CTAs per SM

__global__ void __launch_bounds__(kRelThreads, kRelInsertCtas)
relabel_insert_kernel(Parts ps, RelTable t, void* __restrict__ out, int64_t* status,
                      const RelSurvey* __restrict__ survey, LaunchPad<8>) {
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  const RelUse use = relabel_use(t, numel, survey);
  // One element per thread and step, its successor's id read ahead: more resident threads are worth
  // more than more elements on their way per thread (33.5 M ids in ordinary slots: 660 us, two elements per
  // thread with twice the registers 1,150; in half-size slots 480).  The 7 CTAs per SM leave 32 registers, and
  // 16 bytes a thread are spilled; it took 492 us before 7 were asked for.
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  long long next = i < numel ? part_elem(ps, sizes, i) : 0;
  // The CTAs of the first wave start a little apart: an id that many elements share is claimed by the first of
  // them and found by the others, instead of being met unclaimed by all (see relabel_enter).  1,048,576 ids, a
  // tenth of them the same: 121 us a call with all at once, 108 with 1 us between the CTAs of an SM, 103 with 2;
  // 300,000 distinct ids take 54 us with 0 and 1, 57 with 2.
  if (blockIdx.x >= kRelSms && blockIdx.x < kRelSms * kRelInsertCtas) __nanosleep(blockIdx.x / kRelSms * 1000);
  for (; i < numel; i += stride) {
    const long long key = next;
    if (i + stride < numel) next = part_elem(ps, sizes, i + stride);
    bool maybe_first;
    uint32_t pos;
    if (use.small.stride == 1) {
      pos = (uint32_t)key;
      maybe_first = __ldcg(use.small.words + pos) > (unsigned)i;
      if (maybe_first) {
        maybe_first = relabel_lowest(pos);
        if (maybe_first) atomicMin(use.small.words + pos, (unsigned)i);
      }
    } else if (use.small.stride == 2) {
      pos = relabel_claim_half(use.small, key, (unsigned)i, status, &maybe_first);
    } else {
      pos = relabel_enter<true>(use.range, key, (unsigned)i, status, &maybe_first);
    }
    store_int(out, ps.is64, i, relabel_pack(pos, maybe_first, ps.is64));
  }
}

// Words and half-size slots are not emptied one by one: the front of the table is filled anew.
__global__ void __launch_bounds__(kRelThreads)
relabel_clear_kernel(RelTable t, int64_t numel, const RelSurvey* __restrict__ survey, LaunchPad<48>) {
  const RelSmall small = relabel_use(t, numel, survey).small;
  if (!small.words) return;
  uint4* dst = reinterpret_cast<uint4*>(small.words);
  const uint64_t n = ((uint64_t)small.n * small.stride + 3) / 4;  // a little beyond: all ones there already
  for (uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (uint64_t)gridDim.x * blockDim.x)
    dst[q] = make_uint4(~0u, ~0u, ~0u, ~0u);
}

// Flags first occurrences, numbers them in input order (look-back over the tiles) and finishes
// everything that can be finished for them: the unique id, the element's own result, and the slot,
// which is emptied for the next call and gets the new id in the same 16-byte store (a later
// candidate of the same id finds no index of its own there).  What is left for the
// remap kernel are the repeats alone, marked as such.  A warp takes 32 * ITEMS consecutive
// elements, 32 at a time, so that every access to the streamed arrays is contiguous; all slot
// reads of a thread are in flight together.
// WORDS: ids below t.n_words have a word instead of a slot, and nothing in slot_of yet; a word is final, and
// stays as it is.  A repeat takes down its first occurrence's index.  The seeds of all hops but the first
// are distinct (they are the hop before's unique ids), so theirs need not be looked at.  What bounds it is random
// reads of the words, from L2.  8,192 seeds 5/10/15 on 10 M nodes, behind the last hop (2.8 M ids, 2.4 M of them
// distinct): 45 us with the new ids written to the words, 35 so; the hop, which reads no word any more before it
// lowers it, 62 -> 55.  (The look-back is 3 of the 45; 5 or 6 CTAs per SM, half the tile, a loop over 592 CTAs: the same.)
template <int ITEMS, bool WORDS>
__global__ void __launch_bounds__(kRelThreads, 4)
relabel_compact_kernel(Parts ps, RelTable t, void* slot_of, void* __restrict__ unique, TileStates st,
                       int64_t* ticket, int64_t* status, int64_t* result, HostPost post, LaunchPad<8>) {
  __shared__ int s_warp_firsts[kRelThreads / 32];
  __shared__ LookbackShared s_look;
  __shared__ int s_tile;
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  constexpr int kTile = kRelThreads * ITEMS;
  const int64_t n_tiles = (numel + kTile - 1) / kTile;
  if (blockIdx.x >= n_tiles) {  // the grid is sized for the largest input the caller allows
    if (numel == 0 && blockIdx.x == 0 && threadIdx.x < 32) {
      if (threadIdx.x == 0) {
        st_relaxed64(result, 0);
        __threadfence();
      }
      __syncwarp();
      if (post.n_words)
        post_to_host(post);
      else if (post.host && threadIdx.x == 0)
        post_note(post, 0, 0);
    }
    return;
  }
  const int tile = take_tile(ticket, &s_tile);  // as many CTAs as tiles are left
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)tile * kTile + (int64_t)warp * (32 * ITEMS) + lane;
  uint32_t pos[ITEMS];
  unsigned first[ITEMS];
  unsigned maybe = 0, is_first = 0;  // one bit per element of this thread
  int64_t id[ITEMS];
  if (WORDS) {
    const int64_t distinct = ps.dev_n0 ? sizes.split : 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int64_t i = base + 32 * j;
      id[j] = i < numel ? part_elem(ps, sizes, i) : 0;
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {  // all reads on their way before anything is done with one
      const int64_t i = base + 32 * j;
      first[j] = t.tag + (unsigned)i;
      if (i >= distinct && i < numel && (uint64_t)id[j] < t.n_words) first[j] = __ldcg(t.words + id[j]);
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int64_t i = base + 32 * j;
      pos[j] = kNoSlot;
      first[j] = i < numel ? first[j] - t.tag : 0xFFFFFFFFu;
      if (i < numel && (uint64_t)id[j] >= t.n_words) {
        bool m;
        pos[j] = relabel_unpack(slot_of, ps.is64, i, &m);
        first[j] = __ldcg(&t.slots[pos[j]].first);  // the smallest index, or already its new id
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int64_t i = base + 32 * j;
      pos[j] = 0;
      if (i < numel) {
        bool m;
        pos[j] = relabel_unpack(slot_of, ps.is64, i, &m);
        maybe |= (unsigned)m << j;
      }
    }
    // only an element the inserting pass did not rule out has to look at its slot; its id is fetched
    // along with it (most are first occurrences), so that nothing waits for it behind the look-back
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      first[j] = 0xFFFFFFFFu;
      id[j] = 0;
      if (maybe >> j & 1u) {
        first[j] = __ldcg(&t.slots[pos[j]].first);
        id[j] = part_elem(ps, sizes, base + 32 * j);
      }
    }
  }
  int before = 0, firsts = 0;  // first occurrences of earlier warps and of this one
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    if (first[j] == (unsigned)(base + 32 * j)) is_first |= 1u << j;
    firsts += __popc(__ballot_sync(0xffffffffu, is_first >> j & 1u));
  }
  if (lane == 0) s_warp_firsts[warp] = firsts;
  __syncthreads();
  int64_t total = 0;
#pragma unroll
  for (int w = 0; w < kRelThreads / 32; ++w) {
    if (w < (int)warp) before += s_warp_firsts[w];
    total += s_warp_firsts[w];
  }
  if (threadIdx.x == 0) lookback_publish(st, tile, total);
  const int64_t prefix = lookback_block(st, tile, total, &s_look, status);
  if (threadIdx.x == 0 && tile == n_tiles - 1) {
    st_relaxed64(result, prefix + total);
    if (post.host && !post.n_words) post_note(post, numel - sizes.split, prefix + total);
  }
  if (post.n_words) {
    __syncthreads();  // every thread's look-back (which may flag a timeout) is over
    if (threadIdx.x < 32) post_when_last(post, n_tiles);
  }
  int64_t row_uid = prefix + before;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int64_t i = base + 32 * j;
    const unsigned row = __ballot_sync(0xffffffffu, is_first >> j & 1u);
    if (is_first >> j & 1u) {
      const int64_t uid = row_uid + __popc(row & ((1u << lane) - 1u));
      store_int(unique, ps.is64, uid, id[j]);
      store_int(slot_of, ps.is64, i, uid);
      if (!WORDS || pos[j] != kNoSlot)
        *reinterpret_cast<uint4*>(t.slots + pos[j]) = make_uint4(~0u, ~0u, (unsigned)uid | kRelNewId, ~0u);
    } else if (WORDS) {
      if (i < numel)
        store_int(slot_of, ps.is64, i,
                  relabel_pack(first[j] & ~kRelNewId, pos[j] != kNoSlot && (first[j] & kRelNewId), ps.is64));
    } else if (maybe >> j & 1u) {
      store_int(slot_of, ps.is64, i, relabel_pack(pos[j], false, ps.is64));
    }
    row_uid += __popc(row);
  }
}

// The same for a surveyed (large) input, in three kernels without a look-back: flag, number the tiles,
// number the flagged elements.  Where first occurrences crowd together, as they do at the start of an
// input with many repeats, a tile is ten times the work of another, and in one kernel every later tile
// waits for it: 449 us for 33.5 M ids (431 with half-size slots, 339 with one long run per CTA),
// 310 in three.
constexpr int kFlagItems = 8;
constexpr int kFlagTile = kRelThreads * kFlagItems, kFlagWords = kFlagTile / 32;
inline int64_t flag_tiles(int64_t numel) { return (numel + kFlagTile - 1) / kFlagTile; }
inline size_t flag_bytes(int64_t numel) {  // a bit per element, then a count per tile
  return (size_t)flag_tiles(numel) * (kFlagWords * sizeof(uint32_t) + sizeof(int)) + sizeof(int);
}

__global__ void __launch_bounds__(kRelThreads, 6)
relabel_flag_kernel(RelTable t, int is64, int64_t numel, void* slot_of, uint32_t* __restrict__ flags,
                    int* __restrict__ counts, const RelSurvey* __restrict__ survey, LaunchPad<16>) {
  __shared__ int s_count[kRelThreads / 32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const RelView view(t, numel, survey);
  const int64_t word0 = (int64_t)blockIdx.x * kFlagWords + warp * kFlagItems;  // of this warp
  const int64_t base = word0 * 32 + lane;
  uint32_t pos[kFlagItems];
  unsigned first[kFlagItems], maybe = 0;
#pragma unroll
  for (int u = 0; u < kFlagItems; ++u) {
    pos[u] = 0;
    if (base + 32 * u < numel) {
      bool m;
      pos[u] = relabel_unpack(slot_of, is64, base + 32 * u, &m);
      maybe |= (unsigned)m << u;
    }
  }
#pragma unroll
  for (int u = 0; u < kFlagItems; ++u) {
    first[u] = 0xFFFFFFFFu;
    if (maybe >> u & 1u) first[u] = view.first(pos[u]);
  }
  int firsts = 0;
#pragma unroll
  for (int u = 0; u < kFlagItems; ++u) {
    const bool is_first = first[u] == (unsigned)(base + 32 * u);
    const unsigned word = __ballot_sync(0xffffffffu, is_first);
    firsts += __popc(word);
    if (lane == 0) flags[word0 + u] = word;
    if (!is_first && (maybe >> u & 1u)) store_int(slot_of, is64, base + 32 * u, relabel_pack(pos[u], false, is64));
  }
  if (lane == 0) s_count[warp] = firsts;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < kRelThreads / 32; ++w) sum += s_count[w];
    counts[blockIdx.x] = sum;
  }
}

// One CTA: counts -> first occurrences ahead of each tile; their number goes to the host.
constexpr int kTotalThreads = 1024;
__global__ void __launch_bounds__(kTotalThreads)
relabel_total_kernel(int* counts, int n_tiles, int64_t* result, HostPost post, LaunchPad<32>) {
  __shared__ int64_t s_sums[32];
  __shared__ int64_t s_total;
  // a thread takes consecutive counts, four at a time (the array is 16-byte aligned and, past the
  // tiles, has room for one more count only)
  const int per = ((n_tiles + kTotalThreads - 1) / kTotalThreads + 3) & ~3, lo = (int)threadIdx.x * per;
  const int hi = lo + per < n_tiles ? lo + per : n_tiles;
  int64_t sum = 0;
#pragma unroll 4
  for (int q = lo; q + 4 <= hi; q += 4) {
    const int4 c = *reinterpret_cast<const int4*>(counts + q);
    sum += c.x + c.y + c.z + c.w;
  }
  for (int q = lo < hi ? lo + ((hi - lo) & ~3) : hi; q < hi; ++q) sum += counts[q];
  int at = (int)block_exclusive_scan(sum, s_sums, &s_total);
#pragma unroll 4
  for (int q = lo; q + 4 <= hi; q += 4) {
    const int4 c = *reinterpret_cast<const int4*>(counts + q);
    *reinterpret_cast<int4*>(counts + q) = make_int4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
    at += c.x + c.y + c.z + c.w;
  }
  for (int q = lo < hi ? lo + ((hi - lo) & ~3) : hi; q < hi; ++q) {
    const int c = counts[q];
    counts[q] = at;
    at += c;
  }
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      counts[n_tiles] = (int)s_total;
      st_relaxed64(result, s_total);
      __threadfence();
    }
    __syncwarp();
    post_to_host(post);
  }
}

__global__ void __launch_bounds__(kRelThreads, 4)
relabel_number_kernel(Parts ps, RelTable t, void* slot_of, void* __restrict__ unique,
                      const uint32_t* __restrict__ flags, const int* __restrict__ before,
                      const RelSurvey* __restrict__ survey, LaunchPad<56>) {
  const int tile_before = before[blockIdx.x];
  if (before[blockIdx.x + 1] == tile_before) return;
  static_assert(kFlagWords == 64, "two words of the tile per lane");
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, full = 0xffffffffu;
  const PartSizes sizes{ps.start[kMaxParts], -1};
  const RelView view(t, sizes.numel, survey);
  const int64_t word0 = (int64_t)blockIdx.x * kFlagWords;
  // every warp adds up the tile's words, two per lane, and takes kFlagItems of them
  const uint2 two = reinterpret_cast<const uint2*>(flags + word0)[lane];
  const int both = __popc(two.x) + __popc(two.y);
  int inc = both;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(full, inc, o);
    if (lane >= (unsigned)o) inc += up;
  }
  const int ahead = inc - both;  // of this lane's first word
  const int64_t base = (word0 + warp * kFlagItems) * 32 + lane;
  uint32_t pos[kFlagItems];
  int64_t id[kFlagItems];
  int uid[kFlagItems];
  unsigned mine = 0;
#pragma unroll
  for (int u = 0; u < kFlagItems; ++u) {
    const int from = (int)(warp * kFlagItems + u) / 2;
    const uint32_t x = __shfl_sync(full, two.x, from), y = __shfl_sync(full, two.y, from);
    const uint32_t word = u & 1 ? y : x;
    uid[u] = tile_before + __shfl_sync(full, ahead, from) + (u & 1 ? __popc(x) : 0) + __popc(word & ((1u << lane) - 1u));
    if (word >> lane & 1u) {
      bool m;
      mine |= 1u << u;
      pos[u] = relabel_unpack(slot_of, ps.is64, base + 32 * u, &m);
      id[u] = part_elem(ps, sizes, base + 32 * u);
    }
  }
#pragma unroll
  for (int u = 0; u < kFlagItems; ++u)
    if (mine >> u & 1u) {
      store_int(unique, ps.is64, uid[u], id[u]);
      store_int(slot_of, ps.is64, base + 32 * u, uid[u]);
      view.number(pos[u], (unsigned)uid[u]);
    }
}

// The repeats: slot -> new id.  First occurrences hold theirs already.
__global__ void __launch_bounds__(kRelThreads)
relabel_remap_kernel(Parts ps, RelTable t, void* out, LaunchPad<24>) {
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  constexpr int U = 2;  // independent slot reads per thread in flight
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < numel; i0 += U * stride) {
    uint32_t pos[U];
    unsigned newid[U];
    bool repeat[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      repeat[u] = false;
      if (i < numel) {
        bool done;
        pos[u] = relabel_unpack(out, ps.is64, i, &done);
        repeat[u] = !done;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (repeat[u]) newid[u] = __ldcg(&t.slots[pos[u]].first) & ~kRelNewId;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (repeat[u]) store_int(out, ps.is64, i0 + u * stride, (int64_t)newid[u]);
  }
}

// The repeats of all hops of a mini-batch with words: first occurrence -> its new id.  Nothing of a hop waits for
// that of the hop before, nor does the host, so one kernel at the end does what three kernels of 3 to 9 us did between
// the hops, every hop with CTAs of its own (all with all hops, one after the other: 13.3 us for the 9.8 of 8,192 seeds
// 5/10/15 on 50,000 nodes).  50 seeds 5/10/15 70 -> 65 us, 1,024 seeds 120 -> 115, 8,192 seeds 292 -> 289, 3/40 97 -> 93.
template <bool IS64>
__global__ void __launch_bounds__(kRelThreads) relabel_repeats_kernel(RelRepeats r, LaunchPad<40>) {
  pdl_prologue();
  using T = typename std::conditional<IS64, unsigned long long, unsigned>::type;
  const T mark = IS64 ? (T)kRelNotFirst64 : (T)kRelNotFirst32;
  T* out = static_cast<T*>(r.out[0]);
  const int64_t* words = r.words;
  int64_t seeds = r.n_seeds;
  unsigned first = 0, end = gridDim.x;
#pragma unroll
  for (int h = 1; h < 8; ++h) {
    if (h >= r.n_hops) break;
    if (blockIdx.x >= r.first_cta[h]) {
      out = static_cast<T*>(r.out[h]);
      words = r.words + h * 8;
      seeds = -1;
      first = r.first_cta[h];
    } else {
      end = min(end, r.first_cta[h]);
    }
  }
  const int64_t numel = (seeds < 0 ? words[3 - 8] : seeds) + words[1];
  constexpr int U = 2;  // reads per thread in flight
  const int64_t stride = (int64_t)(end - first) * kRelThreads;
  for (int64_t i0 = (int64_t)(blockIdx.x - first) * kRelThreads + threadIdx.x; i0 < numel; i0 += U * stride) {
    T raw[U], uid[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      raw[u] = 0;
      if (i0 + u * stride < numel) raw[u] = __ldcg(out + i0 + u * stride);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (raw[u] & mark) uid[u] = __ldcg(out + (raw[u] & ~mark));
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (raw[u] & mark) out[i0 + u * stride] = uid[u];
  }
}

int launch_relabel_repeats(RelRepeats r, const int64_t* numel_bounds, bool is64, cudaStream_t s) {
  const int64_t most = (int64_t)sm_count() * 16;
  unsigned ctas = 0;
  for (int h = 0; h < r.n_hops; ++h) {
    r.first_cta[h] = ctas;
    const int64_t want = (numel_bounds[h] + kRelThreads - 1) / kRelThreads;
    ctas += (unsigned)(want < most ? want : most);
  }
  SHMT_CUDA_TRY(launch_kernel(true, is64 ? relabel_repeats_kernel<true> : relabel_repeats_kernel<false>, ctas, kRelThreads,
                              0, s, r, LaunchPad<40>{}));
  return SHMT_OK;
}

// The same for a surveyed input.
__global__ void __launch_bounds__(kRelThreads, 8)
relabel_remap_large_kernel(RelTable t, int is64, int64_t numel, void* out, const RelSurvey* __restrict__ survey,
                           LaunchPad<32>) {
  const RelView view(t, numel, survey);
  constexpr int U = 2;  // 33.5 M ids: 8 reads per thread (5 CTAs) 354 us, 4 (6 CTAs) 232, 2 (8 CTAs) 187, 1 200
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < numel; i0 += U * stride) {
    uint32_t pos[U];
    unsigned newid[U];
    bool repeat[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      repeat[u] = false;
      if (i < numel) {
        bool done;
        pos[u] = relabel_unpack(out, is64, i, &done);
        repeat[u] = !done;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (repeat[u]) newid[u] = view.newid(pos[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (repeat[u]) store_int(out, is64, i0 + u * stride, (int64_t)newid[u]);
  }
}

// Up to kRelSmallMax ids: everything in one CTA, whose table lies in shared memory, instead of three
// kernels that each wait for the one before (and a memset).  What bounds it is latency: one read of
// the ids, a few shared-memory steps, one write.  A call with 800 ids: 36 us with the memset and three
// kernels, 27 so; with 4,096 ids 36 and 31; with 8,192 distinct ids one CTA would take longer (46
// against 39).
constexpr int kRelSmallThreads = 1024;
constexpr int64_t kRelSmallMax = 4096;
static size_t rel_small_smem(uint32_t slots) { return (size_t)slots * (sizeof(long long) + sizeof(unsigned)); }

template <int ITEMS>
__global__ void __launch_bounds__(kRelSmallThreads)
relabel_small_kernel(Parts ps, uint32_t slots, void* __restrict__ unique, void* __restrict__ out, int64_t* status,
                     int64_t* result, HostPost post, LaunchPad<48>) {
  constexpr int kWarps = kRelSmallThreads / 32;
  extern __shared__ __align__(16) unsigned char s_table[];
  long long* s_key = reinterpret_cast<long long*>(s_table);
  unsigned* s_first = reinterpret_cast<unsigned*>(s_key + slots);  // smallest index of the id; later its new id
  __shared__ int s_count[ITEMS * kWarps];
  __shared__ int s_found;
  const unsigned full = 0xffffffffu;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const PartSizes sizes{ps.start[kMaxParts], -1};
  const int numel = (int)sizes.numel;
  const uint32_t mask = slots - 1;
  long long id[ITEMS];
  uint32_t pos[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kRelSmallThreads + tid;
    id[j] = i < numel ? part_elem(ps, sizes, i) : 0;
  }
  for (uint32_t q = (uint32_t)tid; q < slots; q += kRelSmallThreads) {
    s_key[q] = kEmptyKey;
    s_first[q] = 0xFFFFFFFFu;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kRelSmallThreads + tid;
    pos[j] = 0;
    if (i >= numel) continue;
    uint32_t at = (uint32_t)(mix64((uint64_t)id[j]) >> 32) & mask;
    while (true) {  // at most half of the slots are ever taken, so an empty one is met
      long long cur = *reinterpret_cast<volatile long long*>(s_key + at);
      if (cur == kEmptyKey)
        cur = (long long)atomicCAS(reinterpret_cast<unsigned long long*>(s_key + at), (unsigned long long)kEmptyKey,
                                   (unsigned long long)id[j]);
      if (cur == kEmptyKey || cur == id[j]) break;
      at = (at + 1) & mask;
    }
    atomicMin(s_first + at, (unsigned)i);
    pos[j] = at;
  }
  __syncthreads();
  unsigned is_first = 0;  // one bit per element of this thread
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kRelSmallThreads + tid;
    if (i < numel && s_first[pos[j]] == (unsigned)i) is_first |= 1u << j;
    const unsigned row = __ballot_sync(full, is_first >> j & 1u);
    if (lane == 0) s_count[j * kWarps + warp] = __popc(row);
  }
  __syncthreads();
  if (warp == 0) {  // first occurrences ahead of each (element row, warp)
    int run = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int c = s_count[j * kWarps + lane];
      int inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(full, inc, o);
        if (lane >= o) inc += up;
      }
      s_count[j * kWarps + lane] = run + inc - c;
      run += __shfl_sync(full, inc, 31);
    }
    if (lane == 0) {
      s_found = run;
      st_relaxed64(status, DEV_OK);
      st_relaxed64(result, run);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const unsigned row = __ballot_sync(full, is_first >> j & 1u);
    if (is_first >> j & 1u) {
      const int uid = s_count[j * kWarps + warp] + __popc(row & ((1u << lane) - 1u));
      store_int(unique, ps.is64, uid, id[j]);
      s_first[pos[j]] = (unsigned)uid;
    }
  }
  __syncthreads();
  if (warp == 0) post_result(post, s_found);  // behind the last barrier: nobody waits for its way to the host
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kRelSmallThreads + tid;
    if (i < numel) store_int(out, ps.is64, i, (int64_t)s_first[pos[j]]);
  }
}

template <int ITEMS>
static int launch_relabel_small(const Parts& ps, void* out_unique, void* out_relabel, int64_t* words,
                                const HostPost& post, cudaStream_t s) {
  uint32_t slots = 64;
  while ((int64_t)slots < 2 * ps.start[kMaxParts]) slots <<= 1;
  static bool configured[64] = {false};
  int dev = 0;
  SHMT_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && !configured[dev]) {
    SHMT_CUDA_TRY(cudaFuncSetAttribute(relabel_small_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)rel_small_smem(2 * ITEMS * kRelSmallThreads)));
    configured[dev] = true;
  }
  SHMT_CUDA_TRY(launch_kernel(false, relabel_small_kernel<ITEMS>, 1u, kRelSmallThreads, rel_small_smem(slots), s, ps,
                              slots, out_unique, out_relabel, words + W_STATUS, words + W_RESULT, post,
                              LaunchPad<48>{}));
  return SHMT_OK;
}

// Table for up to `numel_bound` ids at load <= 0.5, in the context's block whose keys and
// first-index words are empty between calls (whatever the capacity, so regions of different
// capacities may overlap freely).
// Small inputs get four times the room (see kRelRoomy).
uint64_t relabel_capacity(int64_t numel_bound) {
  uint64_t cap = 64;
  while (cap < (uint64_t)numel_bound * 2) cap <<= 1;
  while (cap < (uint64_t)numel_bound * 8 && cap < (uint64_t)kRelRoomy) cap <<= 1;
  return cap;
}

// Where a call of `numel` ids keeps what: look-back descriptors, or, when it is surveyed, the survey and
// the flags behind it.
struct RelScratch {
  bool look;           // a table that fits the L2 cache gains nothing from compact slots; a larger one may
  size_t zeroed;       // bytes that start at zero; the survey lies behind `states` of them
  size_t states, all;
};
static RelScratch relabel_scratch(int64_t numel) {
  RelScratch r{};
  if (numel <= kRelSmallMax) return r;  // one CTA, all in shared memory
  const int64_t n_tiles = (numel + kRelTile - 1) / kRelTile;
  r.look = relabel_capacity(numel) * sizeof(RelSlot) > kRelSurveyMinTableBytes;
  r.states = (tile_state_bytes(n_tiles) + 255) & ~(size_t)255;
  r.zeroed = r.look ? r.states + sizeof(RelSurvey) : tile_state_bytes(n_tiles);
  r.all = r.zeroed + (r.look ? flag_bytes(numel) : 0);
  return r;
}
size_t relabel_scratch_bytes(int64_t numel) { return relabel_scratch(numel).all; }

int relabel_table(shmt_ctx* ctx, int64_t numel_bound, RelTable* t, cudaStream_t s, const RelWords& words) {
  const uint64_t cap = relabel_capacity(numel_bound);
  if (int rc = ctx_reserve_table(ctx, cap * sizeof(RelSlot), s)) return rc;
  t->slots = reinterpret_cast<RelSlot*>(ctx->table);
  t->cap = (uint32_t)cap;
  t->words = words.n ? ctx->words : nullptr;
  t->n_words = (uint32_t)words.n;
  t->tag = words.tag;
  return SHMT_OK;
}

int launch_relabel(shmt_ctx* ctx, const Parts& ps, int64_t numel_bound, void* out_unique, void* out_relabel, TileStates st, int64_t* ticket,
                   int64_t* status, int64_t* result, cudaStream_t s, bool inserted, bool pdl,
                   const HostPost* post, RelSurvey* survey, const RelWords& words) {
  RelTable t;
  if (int rc = relabel_table(ctx, numel_bound, &t, s, words)) return rc;
  const int64_t n_tiles = (numel_bound + kRelTile - 1) / kRelTile;
  int64_t blocks = (numel_bound + kRelThreads - 1) / kRelThreads;
  const int64_t cap_blocks = (int64_t)sm_count() * 16;
  const unsigned grid = (unsigned)(blocks < cap_blocks ? blocks : cap_blocks);
  if (!inserted) {
    if (survey) SHMT_CUDA_TRY(launch_kernel(pdl, relabel_survey_kernel, grid, kRelThreads, 0, s, ps, survey, LaunchPad<56>{}));
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_insert_kernel, grid, kRelThreads, 0, s, ps, t, out_relabel, status,
                                (const RelSurvey*)survey, LaunchPad<8>{}));
  }
  if (survey) {
    const int64_t tiles = flag_tiles(numel_bound);  // surveyed inputs are of that size exactly
    uint32_t* flags = reinterpret_cast<uint32_t*>(survey + 1);
    int* counts = reinterpret_cast<int*>(flags + tiles * kFlagWords);
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_flag_kernel, (unsigned)tiles, kRelThreads, 0, s, t, ps.is64, numel_bound,
                                out_relabel, flags, counts, (const RelSurvey*)survey, LaunchPad<16>{}));
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_total_kernel, 1u, kTotalThreads, 0, s, counts, (int)tiles, result,
                                post ? *post : HostPost{}, LaunchPad<32>{}));
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_number_kernel, (unsigned)tiles, kRelThreads, 0, s, ps, t, out_relabel,
                                out_unique, (const uint32_t*)flags, (const int*)counts, (const RelSurvey*)survey, LaunchPad<56>{}));
  } else {
    const bool big = numel_bound >= kRelLargeInput;
    const int64_t big_tiles = (numel_bound + kRelThreads * kRelItemsLarge - 1) / (kRelThreads * kRelItemsLarge);
    auto kernel = big ? (words.n ? relabel_compact_kernel<kRelItemsLarge, true> : relabel_compact_kernel<kRelItemsLarge, false>)
                      : (words.n ? relabel_compact_kernel<kRelItems, true> : relabel_compact_kernel<kRelItems, false>);
    SHMT_CUDA_TRY(launch_kernel(pdl, kernel, (unsigned)(big ? big_tiles : n_tiles), kRelThreads, 0, s, ps, t, out_relabel,
                                out_unique, st, ticket, status, result, post ? *post : HostPost{}, LaunchPad<8>{}));
  }
  if (words.n) {
    // launch_relabel_repeats, for all hops at once
  } else if (!survey) {
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_remap_kernel, grid, kRelThreads, 0, s, ps, t, out_relabel, LaunchPad<24>{}));
  } else {
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_remap_large_kernel, grid, kRelThreads, 0, s, t, ps.is64, numel_bound,
                                out_relabel, (const RelSurvey*)survey, LaunchPad<32>{}));
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_clear_kernel, grid, kRelThreads, 0, s, t, numel_bound,
                                (const RelSurvey*)survey, LaunchPad<48>{}));
  }
  SHMT_CUDA_TRY(cudaGetLastError());
  return SHMT_OK;
}

}  // namespace shmt

using namespace shmt;

extern "C" int shmt_relabel(shmt_ctx* ctx, const void* const* parts, const int64_t* part_sizes,
                            int n_parts, int dtype, void* out_unique, void* out_relabel,
                            int64_t* n_unique_host, void* stream) {
  SHMT_REQUIRE(ctx != nullptr, "shmt_relabel: ctx is null");
  SHMT_REQUIRE(valid_int_dtype(dtype), "shmt_relabel: ids can only be int32 or int64");
  SHMT_REQUIRE(n_parts >= 0 && n_parts <= kMaxParts, "shmt_relabel: 0..%d parts", kMaxParts);
  SHMT_REQUIRE(n_parts == 0 || (parts && part_sizes), "shmt_relabel: parts/part_sizes are null");
  Parts ps{};
  ps.n = n_parts;
  ps.is64 = dtype == SHMT_I64;
  int64_t numel = 0;
  for (int p = 0; p < n_parts; ++p) {
    SHMT_REQUIRE(part_sizes[p] >= 0, "shmt_relabel: part %d has negative size", p);
    SHMT_REQUIRE(part_sizes[p] == 0 || parts[p] != nullptr, "shmt_relabel: part %d is null", p);
    ps.ptr[p] = parts[p];
    ps.start[p] = numel;
    numel += part_sizes[p];
  }
  for (int p = n_parts; p <= kMaxParts; ++p) ps.start[p] = numel;
  SHMT_REQUIRE(numel < ((int64_t)1 << 30), "shmt_relabel: %lld ids is too many (limit 2^30)",
               (long long)numel);
  if (numel == 0) {
    if (n_unique_host) *n_unique_host = 0;
    return SHMT_OK;
  }
  SHMT_REQUIRE(out_unique && out_relabel, "shmt_relabel: outputs are null");
  DeviceGuard guard(ctx->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (numel <= kRelSmallMax) {
    // no scratch but the result words, and nothing behind the post that the host has to wait for
    int64_t* w = ctx->d_words();
    HostPost post{};
    if (n_unique_host) post = ctx_begin_post(ctx, w, 4, nullptr);
    int rc = SHMT_OK;
    if (numel <= kRelSmallThreads)
      rc = launch_relabel_small<1>(ps, out_unique, out_relabel, w, post, s);
    else if (numel <= 2 * kRelSmallThreads)
      rc = launch_relabel_small<2>(ps, out_unique, out_relabel, w, post, s);
    else
      rc = launch_relabel_small<4>(ps, out_unique, out_relabel, w, post, s);
    if (rc || !n_unique_host) return rc;
    if (int rc2 = ctx_await_post(ctx, post, s)) return rc2;
    *n_unique_host = ctx->h_words[W_RESULT];
    return SHMT_OK;
  }
  const RelScratch at = relabel_scratch(numel);
  if (int rc = ctx_reserve(ctx, at.all, s)) return rc;
  TileStates st = carve_tile_states(ctx->region(), (numel + kRelTile - 1) / kRelTile);
  RelSurvey* survey = at.look ? reinterpret_cast<RelSurvey*>(ctx->region() + at.states) : nullptr;
  // result words, tile descriptors and the survey to zero
  SHMT_CUDA_TRY(cudaMemsetAsync(ctx->scratch, 0, 256 + at.zeroed, s));
  int64_t* w = ctx->d_words();
  // with a count to return, the compact kernel posts it and the call returns while the remap
  // kernel runs; the next user of the context waits for that kernel first
  HostPost post{};
  if (n_unique_host) post = ctx_begin_post(ctx, w, 4, w + W_DONE);
  if (int rc = launch_relabel(ctx, ps, numel, out_unique, out_relabel, st, w + W_TICKET,
                              w + W_STATUS, w + W_RESULT, s, false, false,
                              n_unique_host ? &post : nullptr, survey))
    return rc;
  if (n_unique_host) {
    if (int rc = ctx_mark_tail(ctx, s)) return rc;
    if (int rc = ctx_await_post(ctx, post, s)) return rc;
    if (int rc = ctx_status_of_words(ctx, "shmt_relabel")) return rc;
    *n_unique_host = ctx->h_words[W_RESULT];
  }
  return SHMT_OK;
}
