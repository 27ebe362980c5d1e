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
// The element counts may live on the device (written by an earlier kernel), so a
// chain of hops can be queued without the host knowing any size.
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
// huge), and how many distinct ids it holds, from a sample.
__global__ void __launch_bounds__(kRelThreads)
relabel_survey_kernel(Parts ps, RelSurvey* survey) {
  __shared__ unsigned s_marked[kRelThreads / 32];
  pdl_prologue();
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
      if (!(__ldcg(survey->bitmap + (at >> 5)) & bit))
        marked += (atomicOr(survey->bitmap + (at >> 5), bit) & bit) == 0;
    }
  };
#pragma unroll
  for (int p = 0; p < kMaxParts; ++p) {
    if (p >= ps.n) break;
    const int64_t n = ps.start[p + 1] - ps.start[p];
    int64_t done = 0;  // elements covered by the 16-byte loads below
    if ((reinterpret_cast<uintptr_t>(ps.ptr[p]) & 15) == 0) {
      // an aligned part: 16-byte loads, four per thread in flight
      const int per = ps.is64 ? 2 : 4;
      const int64_t n_vec = n / per;
      const uint4* src = static_cast<const uint4*>(ps.ptr[p]);
      for (int64_t v = gtid; v < n_vec; v += 4 * stride) {
        uint4 x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (v + u * stride < n_vec) x[u] = __ldg(src + v + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
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
    if (m) atomicMax(&survey->largest, m);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    marked = 0;
    for (int w = 0; w < kRelThreads / 32; ++w) marked += s_marked[w];
    if (marked) atomicAdd(&survey->marked, (unsigned long long)marked);
  }
}

// How a call of `numel` ids uses the table.  Without a survey: at least two slots per id, as if all
// were distinct.  With one: ids that all fit the table are their own slots (a frontier of densely
// numbered nodes touches a compact part of the table); else kRelSlotsPerId slots per distinct id.
constexpr double kRelSlotsPerId = 2.0;
__device__ __forceinline__ RelRange relabel_range(const RelTable& t, int64_t numel, const RelSurvey* survey) {
  RelRange r{t.slots, relabel_near((double)numel, relabel_slots_per_id((double)numel, 2.0), t.cap), t.cap, false};
  if (survey) {
    if (survey->largest < (unsigned long long)t.cap) {
      r.near = t.cap;
      r.direct = true;
    } else {
      const float bits = (float)(1 << kRelSampleBits), free_bits = bits - (float)survey->marked;
      const float sampled = free_bits > 0.0f ? -bits * logf(free_bits / bits) : bits * 16.0f;
      const double ids = (double)sampled * (double)(1ull << relabel_sample_shift(numel));
      r.near = relabel_near(ids < (double)numel ? ids : (double)numel, kRelSlotsPerId, t.cap);
    }
  }
  return r;
}

__global__ void __launch_bounds__(kRelThreads, 6)
relabel_insert_kernel(Parts ps, RelTable t, void* __restrict__ out, int64_t* status,
                      const RelSurvey* __restrict__ survey) {
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  const RelRange range = relabel_range(t, numel, survey);
  // One element per thread and step, its successor's id read ahead: eight resident CTAs of 32
  // registers claim 33.5 M ids in 660 us where two elements per thread (80 registers) took 1,150.
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  long long next = i < numel ? part_elem(ps, sizes, i) : 0;
  for (; i < numel; i += stride) {
    const long long key = next;
    if (i + stride < numel) next = part_elem(ps, sizes, i + stride);
    unsigned seen;
    const uint32_t pos = relabel_claim(range, key, status, &seen);
    store_int(out, ps.is64, i, relabel_pack(pos, relabel_settle(range, pos, seen, (unsigned)i), ps.is64));
  }
}

// Flags first occurrences, numbers them in input order (look-back over the tiles) and finishes
// everything that can be finished for them: the unique id, the element's own result, and the slot,
// which gets the new id and is emptied for the next call in the same 16-byte store (a later
// candidate of the same id still finds an index that is not its own there).  What is left for the
// remap kernel are the repeats alone, marked as such.  A warp takes 32 * ITEMS consecutive
// elements, 32 at a time, so that every access to the streamed arrays is contiguous; all slot
// reads of a thread are in flight together.
template <int ITEMS>
__global__ void __launch_bounds__(kRelThreads, 4)
relabel_compact_kernel(Parts ps, RelTable t, void* slot_of, void* __restrict__ unique, TileStates st,
                       int64_t* ticket, int64_t* status, int64_t* result, HostPost post) {
  __shared__ int s_warp_firsts[kRelThreads / 32];
  __shared__ LookbackShared s_look;
  __shared__ int s_tile;
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  constexpr int kTile = kRelThreads * ITEMS;
  const int64_t n_tiles = (numel + kTile - 1) / kTile;
  const int tile = take_tile(ticket, &s_tile);
  if (tile >= n_tiles) {  // the grid is sized for the largest input the caller allows
    if (numel == 0 && tile == 0 && threadIdx.x < 32) {
      if (threadIdx.x == 0) {
        st_relaxed64(result, 0);
        __threadfence();
      }
      __syncwarp();
      post_to_host(post);
    }
    return;
  }
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)tile * kTile + (int64_t)warp * (32 * ITEMS) + lane;
  uint32_t pos[ITEMS];
  unsigned first[ITEMS];
  unsigned maybe = 0, is_first = 0;  // one bit per element of this thread
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
  // only an element the inserting pass did not rule out has to look at its slot
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    first[j] = 0xFFFFFFFFu;
    if (maybe >> j & 1u) first[j] = __ldcg(&t.slots[pos[j]].first);
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
  if (threadIdx.x == 0 && tile == n_tiles - 1) st_relaxed64(result, prefix + total);
  if (post.host) {
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
      store_int(unique, ps.is64, uid, part_elem(ps, sizes, i));
      store_int(slot_of, ps.is64, i, uid);
      *reinterpret_cast<uint4*>(t.slots + pos[j]) = make_uint4(~0u, ~0u, ~0u, (unsigned)uid);
    } else if (maybe >> j & 1u) {
      store_int(slot_of, ps.is64, i, relabel_pack(pos[j], false, ps.is64));
    }
    row_uid += __popc(row);
  }
}

// The repeats: slot -> new id.  First occurrences hold theirs already.
__global__ void __launch_bounds__(kRelThreads)
relabel_remap_kernel(Parts ps, RelTable t, void* out) {
  pdl_prologue();
  const PartSizes sizes = resolve_sizes(ps);
  const int64_t numel = sizes.numel;
  constexpr int U = 4;  // independent slot reads per thread in flight
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
      if (repeat[u]) newid[u] = __ldcg(&t.slots[pos[u]].newid);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (repeat[u]) store_int(out, ps.is64, i0 + u * stride, (int64_t)newid[u]);
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
                     int64_t* result, HostPost post) {
  constexpr int kWarps = kRelSmallThreads / 32;
  extern __shared__ __align__(16) unsigned char s_table[];
  long long* s_key = reinterpret_cast<long long*>(s_table);
  unsigned* s_first = reinterpret_cast<unsigned*>(s_key + slots);  // smallest index of the id; later its new id
  __shared__ int s_count[ITEMS * kWarps];
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
  if (warp == 0) post_to_host(post);  // behind the last barrier: nobody waits for its way to the host
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
  relabel_small_kernel<ITEMS><<<1, kRelSmallThreads, rel_small_smem(slots), s>>>(
      ps, slots, out_unique, out_relabel, words + W_STATUS, words + W_RESULT, post);
  SHMT_CUDA_TRY(cudaGetLastError());
  return SHMT_OK;
}

// Table for up to `numel_bound` ids at load <= 0.5, in the context's block whose keys and
// first-index words are all ones between calls (whatever the capacity, so regions of different
// capacities may overlap freely); the new-id words need no initial value.
// Small inputs get four times the room (see kRelRoomy).
uint64_t relabel_capacity(int64_t numel_bound) {
  uint64_t cap = 64;
  while (cap < (uint64_t)numel_bound * 2) cap <<= 1;
  while (cap < (uint64_t)numel_bound * 8 && cap < (uint64_t)kRelRoomy) cap <<= 1;
  return cap;
}

int relabel_table(shmt_ctx* ctx, int64_t numel_bound, RelTable* t, cudaStream_t s) {
  const uint64_t cap = relabel_capacity(numel_bound);
  if (int rc = ctx_reserve_table(ctx, cap * sizeof(RelSlot), s)) return rc;
  t->slots = reinterpret_cast<RelSlot*>(ctx->table);
  t->cap = (uint32_t)cap;
  return SHMT_OK;
}

int launch_relabel(shmt_ctx* ctx, const Parts& ps, int64_t numel_bound, void* out_unique, void* out_relabel, TileStates st, int64_t* ticket,
                   int64_t* status, int64_t* result, cudaStream_t s, bool inserted, bool pdl,
                   const HostPost* post, RelSurvey* survey) {
  RelTable t;
  if (int rc = relabel_table(ctx, numel_bound, &t, s)) return rc;
  const int64_t n_tiles = (numel_bound + kRelTile - 1) / kRelTile;
  int64_t blocks = (numel_bound + kRelThreads - 1) / kRelThreads;
  const int64_t cap_blocks = (int64_t)sm_count() * 16;
  const unsigned grid = (unsigned)(blocks < cap_blocks ? blocks : cap_blocks);
  if (!inserted) {
    if (survey) SHMT_CUDA_TRY(launch_kernel(pdl, relabel_survey_kernel, grid, kRelThreads, 0, s, ps, survey));
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_insert_kernel, grid, kRelThreads, 0, s, ps, t, out_relabel, status,
                                (const RelSurvey*)survey));
  }
  if (numel_bound >= kRelLargeInput) {
    const int64_t big_tiles = (numel_bound + kRelThreads * kRelItemsLarge - 1) / (kRelThreads * kRelItemsLarge);
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_compact_kernel<kRelItemsLarge>, (unsigned)big_tiles, kRelThreads, 0, s,
                                ps, t, out_relabel, out_unique, st, ticket, status, result,
                                post ? *post : HostPost{}));
  } else {
    SHMT_CUDA_TRY(launch_kernel(pdl, relabel_compact_kernel<kRelItems>, (unsigned)n_tiles, kRelThreads, 0, s, ps, t,
                                out_relabel, out_unique, st, ticket, status, result,
                                post ? *post : HostPost{}));
  }
  SHMT_CUDA_TRY(launch_kernel(pdl, relabel_remap_kernel, grid, kRelThreads, 0, s, ps, t, out_relabel));
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
  const int64_t n_tiles = (numel + kRelTile - 1) / kRelTile;
  const size_t states = (tile_state_bytes(n_tiles) + 255) & ~(size_t)255;
  // a table that fits the L2 cache gains nothing from compact slots; a larger one may
  const bool look = relabel_capacity(numel) * sizeof(RelSlot) > kRelSurveyMinTableBytes;
  const size_t zeroed = look ? states + sizeof(RelSurvey) : tile_state_bytes(n_tiles);
  if (int rc = ctx_reserve(ctx, zeroed)) return rc;
  TileStates st = carve_tile_states(ctx->region(), n_tiles);
  RelSurvey* survey = look ? reinterpret_cast<RelSurvey*>(ctx->region() + states) : nullptr;
  // result words, tile descriptors and the survey to zero
  SHMT_CUDA_TRY(cudaMemsetAsync(ctx->scratch, 0, 256 + zeroed, s));
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
