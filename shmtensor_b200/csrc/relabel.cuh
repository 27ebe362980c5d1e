// Shared declarations of the relabel kernels (used by relabel.cu and the fused
// multi-hop sampler).
#pragma once

#include "ctx.cuh"
#include "lookback.cuh"

namespace shmt {

constexpr int kRelThreads = 256;
// Elements per thread of the compact kernel, and so per tile.  Grids for kRelLargeInput elements and
// more use kRelItemsLarge per thread (behind a hop of 1.5 M edges: 61 us with 4, 54 with 8, 57 with
// 16); a small input is a few dependent reads long and wants many CTAs.  Look-back state is always
// sized for the small tile.
constexpr int kRelItems = 4;
constexpr int kRelItemsLarge = 8;
constexpr int64_t kRelLargeInput = 4 << 20;
constexpr int kRelTile = kRelThreads * kRelItems;
constexpr int kMaxParts = 8;

struct Parts {
  const void* ptr[kMaxParts];
  int64_t start[kMaxParts + 1];  // element offset of each part; start[kMaxParts] = total
  int n;
  int is64;
  // Two-part form whose sizes were produced on the device (dev_n1 set): |part 1| = *dev_n1,
  // |part 0| = *dev_n0, or the host's start[1] if dev_n0 is null.  start[] stays as the host left it: the
  // kernels keep the sizes they read beside the parts (PartSizes in relabel.cu).
  const int64_t* dev_n0;
  const int64_t* dev_n1;
};

// One 16-byte slot per distinct id, so that claiming the key and recording the first occurrence
// touch one sector, as do reading the new id and emptying the slot.  The new id takes the place of
// `first`, marked so that it is larger than any index: it needs no clearing for the next call.
struct __align__(16) RelSlot {
  long long key;    // -1 = empty
  unsigned first;   // smallest input index holding the key; kRelNewId and more: none yet
  unsigned unused;  // all ones, always
};
constexpr unsigned kRelNewId = 0x80000000u;  // indexes and new ids stay below 2^30

// Mini-batches on a graph of up to kRelMaxWords nodes: a word per node, the smallest index of that id in the hop,
// plus the hop's `tag`.  An id below `n_words` is its own position and nothing has to be claimed: a minimum, which
// nobody waits for, where a slot takes a 32-byte read, a compare-and-swap and a minimum; and the words
// of a graph fit the L2 cache where the slots of a large frontier do not.  Tags go down from hop to hop by
// as many numbers as it can have indices, so that whatever earlier hops have left is larger than all of this
// one's, and no word is ever put back (but all of them when the tags have come down, every 429 batches of
// 10 M ids).  An element that finds another's index in its word is a repeat of that element, whose result it takes.
// Other ids (a last hop may reach nodes that have no row) take slots.
// Slots against words, 5/10/15, 5 to 35 neighbours drawn evenly: 8,192 seeds, 2.4 M nodes 478 us and 317, 10 M 674 and 345,
// 24 M 731 and 454, 33 M 751 and 481; 1,024 seeds 153 and 123, 158 and 130, 158 and 142, 158 and 146; 50 seeds 74 to 80 and 65
// to 74.  The line is at 128 MB of words, about the L2 cache, for each stream that samples; beyond it the gain shrinks (3 to
// 17 neighbours, int32, 8,192 seeds: 50 M nodes 433 and 361, 110 M 436 and 409; 1,024 seeds 128 and 118, 128 and
// 126) while the memory grows to 200 and 440 MB a stream.
struct RelTable {
  RelSlot* slots;  // cap entries
  uint32_t cap;
  uint32_t n_words;
  unsigned* words;  // n_words entries; nullptr: none
  unsigned tag;
};
constexpr int64_t kRelMaxWords = 1 << 25;

// Slots per id.  A small input waits for its longest walk (at half load a few of 5,000 ids walk six
// pairs, 1 us each), so it spreads out over up to kRelRoomy slots; a large one is bound by the
// sectors it draws from HBM and stays compact.  The price is memory: a context that serves 300,000 ids
// holds 48 MB of table where two slots per id would be 24.
constexpr double kRelRoomy = (double)(1 << 21);  // 32 MB

// What a first look at a large input says about it.
constexpr int kRelSampleBits = 20;  // size of the bitmap that counts the distinct ids of the sample
struct RelSurvey {
  unsigned long long largest;  // largest id, read as an unsigned number
  unsigned long long marked;   // bits set in the bitmap
  uint32_t bitmap[1 << (kRelSampleBits - 5)];
};

#ifdef __CUDACC__
// What the inserting pass leaves per element in the output array: the element's slot, plus a mark
// on the elements that are certainly NOT the first occurrence of their id (they met a smaller index
// in the slot), so that the later passes need not look at the slot to know.  The compact kernel
// turns this into: no mark = the element is a first occurrence and holds its new id already;
// mark = a repeat, whose new id is in the slot.  A 32-bit array has room for the mark because the
// table never has more than 2^31 slots (inputs stay below 2^30 ids).
constexpr unsigned long long kRelNotFirst64 = 1ull << 40;
constexpr uint32_t kRelNotFirst32 = 0x80000000u;
// With words, a repeat is marked and holds its first occurrence's index.

__device__ __forceinline__ int64_t relabel_pack(uint32_t pos, bool unmarked, bool is64) {
  if (is64) return (int64_t)((unsigned long long)pos | (unmarked ? 0ull : kRelNotFirst64));
  return (int64_t)(int32_t)(unmarked ? pos : pos | kRelNotFirst32);
}

__device__ __forceinline__ uint32_t relabel_unpack(const void* slot_of, bool is64, int64_t i, bool* unmarked) {
  if (is64) {
    const unsigned long long raw = reinterpret_cast<const unsigned long long*>(slot_of)[i];
    *unmarked = !(raw & kRelNotFirst64);
    return (uint32_t)raw;
  }
  const uint32_t raw = reinterpret_cast<const uint32_t*>(slot_of)[i];
  *unmarked = !(raw & kRelNotFirst32);
  return raw & ~kRelNotFirst32;
}

// The part of the table one call uses.  A key is looked for in consecutive slots from its home in
// [0, near) on, and after kRelNearProbes slots from a second home in [near, full); every element of
// a call walks the same way, so `near` may be smaller than the distinct ids need: it decides how
// compact the used slots lie (what fits the L2 cache is never read from HBM), not whether they fit.
// Homes are even and slots are read in pairs, 32 bytes and one sector a time: at half load the home
// pair is full of other keys for 1 id in 12, where a single slot is taken for 1 in 3, and a warp
// waits for the lane that walks furthest.
struct RelRange {
  RelSlot* slots;
  uint32_t near, full;  // even
};
constexpr uint32_t kRelNearProbes = 128;

// `near` for about `ids` distinct ids at `per_id` slots each.  What little the rest would hold if
// `near` took most of the table is not worth a second region.
__device__ __forceinline__ uint32_t relabel_near(double ids, double per_id, uint32_t full) {
  double want = ids * per_id;
  if (want < 8.0 * kRelNearProbes) want = 8.0 * kRelNearProbes;  // never a lap before the second region
  if (want >= 0.5 * (double)full) return full;
  return (uint32_t)want & ~1u;
}

__device__ __forceinline__ double relabel_slots_per_id(double ids, double least) {
  return ids * least >= kRelRoomy ? least : (ids * 8.0 <= kRelRoomy ? 8.0 : kRelRoomy / ids);
}

struct RelPair {
  long long key0, key1;
  unsigned first0, first1;
};
// Slots at, at + 1 (`at` even), past L1: other CTAs' claims are made in L2.
__device__ __forceinline__ RelPair relabel_load_pair(const RelSlot* slots, uint32_t at) {
  unsigned long long k0, m0, k1, m1;
  asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(k0), "=l"(m0), "=l"(k1), "=l"(m1)
               : "l"(slots + at)
               : "memory");
  return RelPair{(long long)k0, (long long)k1, (unsigned)m0, (unsigned)m1};
}

__device__ __forceinline__ long long relabel_cas(RelSlot* slot, long long key) {
  return (long long)atomicCAS(reinterpret_cast<unsigned long long*>(&slot->key), (unsigned long long)kEmptyKey,
                              (unsigned long long)key);
}

__device__ __forceinline__ uint32_t relabel_home(const RelRange& t, long long key) {
  return __umulhi((uint32_t)(mix64((uint64_t)key) >> 32), t.near) & ~1u;
}

// The slot behind `at` on the way of `key`.
__device__ __forceinline__ uint32_t relabel_next(const RelRange& t, long long key, uint32_t at) {
  ++at;
  if (at & 1u) return at;  // the other slot of a pair
  if (at <= t.near) {
    if (t.near < t.full) {
      const uint32_t home = relabel_home(t, key), walked = at > home ? at - home : at + t.near - home;
      if (walked >= kRelNearProbes) return t.near + (__umulhi((uint32_t)mix64((uint64_t)key), t.full - t.near) & ~1u);
    }
    return at == t.near ? 0u : at;
  }
  return at == t.full ? t.near : at;
}

// Whether the calling lane is the lowest, of those that call together, with its `at`.
__device__ __forceinline__ bool relabel_lowest(uint32_t at) {
  return __ffs(__match_any_sync(__activemask(), at)) - 1 == (int)(threadIdx.x & 31);
}

// Claim (or find) the slot of `key` and enter index `i` for it as a candidate first occurrence;
// *maybe_first is false if it certainly is not one.
// What bounds this is latency: a read of the home, then a CAS if it had room, 0.7 - 1 us each and more under
// load.  `first` only ever goes down: when the index seen there is already smaller than this one the
// atomic would change nothing, and most elements of a frontier are such repeats.  Nothing waits for
// the atomic's result: an element that lowers the index, or loses to a still smaller one, is simply left
// among the candidates.
// CROWDED: an id that many elements share is met unclaimed by every warp on its way when the call starts, and
// atomics on one address are served one after the other (1,048,576 ids, a tenth of them the same: 146 us a
// call, 108 so).  The lanes of a warp that are about to change the same slot leave it to the lowest of them
// (indexes go up with the lanes), and one that lost its claim to another warp looks at the index once more
// first.  A sampling hop, whose warps arrive spread out by their reads of the graph, is better without (8,192 seeds
// 5/10/15 on a graph whose neighbours crowd: 161 us for 164).
template <bool CROWDED>
__device__ __forceinline__ uint32_t relabel_enter(const RelRange& t, long long key, unsigned i, int64_t* status,
                                                  bool* maybe_first) {
  uint32_t pos = relabel_home(t, key);
  for (uint32_t round = 0;; ++round) {
    const RelPair p = relabel_load_pair(t.slots, pos & ~1u);
    const bool second = (pos & 1u) || (p.key0 != key && p.key0 != kEmptyKey);
    const long long cur = second ? p.key1 : p.key0;
    pos |= (uint32_t)second;
    if (cur == key) {
      *maybe_first = (second ? p.first1 : p.first0) > i;  // a mark counts as no index
      if (CROWDED && *maybe_first) *maybe_first = relabel_lowest(pos);
      if (*maybe_first) atomicMin(&t.slots[pos].first, i);
      return pos;
    }
    if (cur == kEmptyKey) {
      // reads next what the lowest lane did: once per lane below this one at most, for the slot is taken then
      if (CROWDED && !relabel_lowest(pos)) continue;
      const long long old = relabel_cas(t.slots + pos, key);
      if (old == kEmptyKey || old == key) {
        *maybe_first = !CROWDED || old == kEmptyKey || *reinterpret_cast<volatile unsigned*>(&t.slots[pos].first) > i;
        if (*maybe_first) atomicMin(&t.slots[pos].first, i);
        return pos;
      }
    }
    if (round > t.full) {  // there are never fewer slots than ids: cannot happen
      atomicMax(reinterpret_cast<unsigned long long*>(status), (unsigned long long)DEV_OVERFLOW);
      *maybe_first = false;
      return pos;
    }
    pos = relabel_next(t, key, pos);
  }
}
#endif

// Slots of the table that serves up to `numel_bound` ids.
uint64_t relabel_capacity(int64_t numel_bound);

// Context scratch that shmt_relabel takes for up to `numel` ids.
size_t relabel_scratch_bytes(int64_t numel);

// Words of a hop (n = 0: none), which ctx_reserve_words has made room for.
struct RelWords {
  int64_t n = 0;
  unsigned tag = 0;
};

// Queue the relabel kernels: insert, compact and remap, or, of a surveyed input, survey, insert, flag,
// total, number, remap and clear.  `numel_bound` >= the real element count sizes the table and the
// grids; ticket/status/result are zeroed device words.
// `pdl`: launch with programmatic stream serialization (see pdl_prologue in common.cuh).
// `inserted`: the slots were already claimed and recorded in out_relabel by the producer
// of the ids (the fused sampling kernel), so only the compact and remap kernels run.
// `post`: the compact (or total) kernel hands the result words to the host as soon as the unique count
// is final; the kernels still to run then produce neither sizes nor errors.
// `words`: what the producer that `inserted` was given.
// `survey`: zeroed device memory, with room for the flags behind it (relabel_scratch_bytes in all); when
// given, a first kernel looks the ids over and the others use the form of the table that suits them
// (see relabel_survey_kernel, relabel_use).
int launch_relabel(shmt_ctx* ctx, const Parts& ps, int64_t numel_bound, void* out_unique, void* out_relabel,
                   TileStates st, int64_t* ticket, int64_t* status, int64_t* result, cudaStream_t s,
                   bool inserted = false, bool pdl = false, const HostPost* post = nullptr,
                   RelSurvey* survey = nullptr, const RelWords& words = {});

// The repeats of the hops of a mini-batch that was relabelled with words: `out` as the compact kernels left it,
// `words` the sizes ([8 h + 1] edges and [8 h + 3] distinct ids of hop h).  launch_relabel leaves them out.
struct RelRepeats {
  void* out[8];
  const int64_t* words;
  int64_t n_seeds;
  int n_hops;
  unsigned first_cta[8];  // of each hop; set by launch_relabel_repeats
};
// `numel_bounds`: most elements of every hop.
int launch_relabel_repeats(RelRepeats r, const int64_t* numel_bounds, bool is64, cudaStream_t s);

// The context's table for `numel_bound` ids (reserving it).
int relabel_table(shmt_ctx* ctx, int64_t numel_bound, RelTable* t, cudaStream_t s, const RelWords& words = {});

}  // namespace shmt
