// Fused probe + row gather (fetch) and probe + row scatter (set / insert-set).
//
// One warp owns a tile of R consecutive requests.  Phase A: one request per
// lane -- load the id, resolve its row address (cooperative map probe, caller's
// mask, or plain host row) and park the address in shared memory.  Phase B: the
// tile's rows are treated as one flat list of VEC-byte chunks that the 32 lanes
// stride through, U chunks per lane in flight before the first is used.  The
// request side of the copy (the output of a fetch, the update of a set) is
// contiguous over the whole tile; the table side jumps from row to row.  All
// lanes stay busy whatever the row size (400-byte rows are 25 chunks, not a
// multiple of 32), and loads that cross the host link or NVLink overlap with
// HBM loads of the same batch.
//
// Replaces the reference's six fetch and six set kernels
// (src/cache_feature_fetch.cu:15-45,89-129,188-224;
//  src/cache_feature_set.cu:6-37,77-116,167-207), which walk 32 rows per warp one
// after another with 4-byte accesses and probe the map redundantly on 32 lanes.
#include <stdlib.h>

#include "bulk.cuh"
#include "ctx.cuh"
#include "kept.h"
#include "map.cuh"

namespace shmt {

constexpr int kRowThreads = 256;
constexpr int kRowWarps = kRowThreads / 32;
constexpr int kMaxBases = 16;

enum : int { MODE_HOST = 0, MODE_MAP = 1, MODE_MASK = 2 };

struct RowJob {
  MapView map;
  const void* mask;
  int mask64;
  int mode;
  char* host;             // host table (UVA) or nullptr
  char* bases[kMaxBases]; // cached-row buffers: [0] local; more for a partitioned cache
  int owner_shift;        // value = (owner << owner_shift) | slot
  const void* idx;
  int idx64;
  int64_t n;
  int64_t row_bytes;
  char* flat;             // fetch: output; set: update rows (request order)
  int rows_per_tile;      // R, 1..32
  LaunchPad<60> pad;
};

template <int VEC> struct VecT;
template <> struct VecT<16> { using type = uint4; };
template <> struct VecT<8> { using type = uint2; };
template <> struct VecT<4> { using type = uint32_t; };
template <> struct VecT<2> { using type = uint16_t; };
template <> struct VecT<1> { using type = uint8_t; };

template <int VEC>
__device__ __forceinline__ typename VecT<VEC>::type load_chunk(const char* p) {
  return __ldg(reinterpret_cast<const typename VecT<VEC>::type*>(p));
}
template <>
__device__ __forceinline__ uint4 load_chunk<16>(const char* p) {
  return ld_stream16(p);
}
template <int VEC>
__device__ __forceinline__ void store_chunk(char* p, typename VecT<VEC>::type v) {
  *reinterpret_cast<typename VecT<VEC>::type*>(p) = v;
}
template <>
__device__ __forceinline__ void store_chunk<16>(char* p, uint4 v) {
  st_stream16(p, v);
}

// Row address of request `first + lane` of a tile (nullptr: nothing to copy).
// All 32 lanes must call: the map probe is cooperative.
__device__ __forceinline__ int64_t load_id(const RowJob& job, int64_t first, int rows,
                                            unsigned lane) {
  return (int)lane < rows ? load_int(job.idx, job.idx64, first + lane) : kEmptyKey;
}

__device__ __forceinline__ char* resolve_row(const RowJob& job, int64_t first, int rows,
                                             unsigned lane, int64_t slot_mask, int64_t id) {
  const bool valid = (int)lane < rows;
  int64_t v = -1;
  if (job.mode == MODE_MAP)
    v = warp_find(job.map, id, valid);
  else if (job.mode == MODE_MASK)
    v = valid ? load_int(job.mask, job.mask64, first + lane) : -1;
  char* p = nullptr;
  if (valid) {
    if (v >= 0) {
      char* base = job.bases[v >> job.owner_shift];
      if (base) p = base + (v & slot_mask) * job.row_bytes;
    } else if (job.host) {
      p = job.host + id * job.row_bytes;
    }
  }
  return p;
}

// The table rows of the tiles a warp goes through, tile0, tile0 + stride, ..., looked up for as many
// tiles as 32 lanes hold rows of, and while the ones before them are still being copied: a tile of 5
// rows would leave 27 lanes of the probe idle and wait for its ids, then for its slots, every time.
// (150,001 rows of 602 bytes: 41 -> 35 us with their lookup.  row_gather_bulk_kernel does without: rows
// that are in L2 gained there, 134 -> 107 us for 1.2 M of 400 bytes, but its usual batches lost, 158 ->
// 177: a steadier stream of reads between its writes is slower in HBM.)
struct RowCursor {
  int64_t tile0, stride, n_tiles;
  int tiles;      // looked up together
  int mine, row;  // the tile of those, and its row, that this lane looks up
  int64_t at;     // first tile (counted along the warp's way) of those in `here`
  char* here;
  char* next;     // of the tiles behind them, once `ready`
  int64_t next_id;
  bool ready;

  __device__ __forceinline__ int64_t index_of(const RowJob& job, int64_t from) const {
    const int64_t tile = tile0 + (from + mine) * stride;
    const int64_t i = tile * job.rows_per_tile + row;
    return mine < tiles && tile < n_tiles && i < job.n ? i : -1;
  }
  __device__ __forceinline__ void fetch_ids(const RowJob& job, int64_t from) {
    const int64_t i = index_of(job, from);
    next_id = i >= 0 ? load_int(job.idx, job.idx64, i) : kEmptyKey;
    ready = false;
  }
  __device__ __forceinline__ void resolve(const RowJob& job, int64_t from, int64_t slot_mask) {
    next = nullptr;
    ready = true;
    if (tile0 + from * stride >= n_tiles) return;  // the same on every lane
    const int64_t i = index_of(job, from);
    int64_t v = -1;
    if (job.mode == MODE_MAP)
      v = warp_find(job.map, next_id, i >= 0);
    else if (job.mode == MODE_MASK)
      v = i >= 0 ? load_int(job.mask, job.mask64, i) : -1;
    if (i >= 0) {
      if (v >= 0) {
        char* base = job.bases[v >> job.owner_shift];
        if (base) next = base + (v & slot_mask) * job.row_bytes;
      } else if (job.host) {
        next = job.host + next_id * job.row_bytes;
      }
    }
  }
  __device__ __forceinline__ RowCursor(const RowJob& job, int64_t first_tile, int64_t stride_, int64_t slot_mask)
      : tile0(first_tile), stride(stride_), at(0) {
    const int lane = (int)(threadIdx.x & 31);
    n_tiles = (job.n + job.rows_per_tile - 1) / job.rows_per_tile;
    tiles = 32 / job.rows_per_tile;
    mine = lane / job.rows_per_tile;
    row = lane % job.rows_per_tile;
    fetch_ids(job, 0);
    resolve(job, 0, slot_mask);
    here = next;
    fetch_ids(job, tiles);
  }
  // The row of this lane in the k-th tile of the warp (nullptr: none); k goes up by one from call to call.
  __device__ __forceinline__ char* row_of(const RowJob& job, int64_t k, int64_t slot_mask) {
    if (k == at + tiles) {
      if (!ready) resolve(job, k, slot_mask);
      here = next;
      at = k;
      fetch_ids(job, k + tiles);
    } else if (k == at + 1) {
      resolve(job, at + tiles, slot_mask);  // its ids have been on their way for a tile
    }
    const int lane = (int)(threadIdx.x & 31);
    const int from = (int)(k - at) * job.rows_per_tile + lane;
    char* p = reinterpret_cast<char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(here), from & 31));
    return lane < job.rows_per_tile ? p : nullptr;
  }
};

// Set by a kernel whose bounded wait ran out; read (and cleared) by shmt_device_fault().
__device__ int g_device_fault = 0;

// Fetch through the TMA unit: rows never pass through registers.  Per warp, a ring
// of STAGES shared-memory buffers of R rows each (about 2 KB): every lane of a tile
// issues one bulk copy (row -> its slot of the buffer) that completes on the stage's
// mbarrier; the whole buffer then leaves with ONE bulk store, because the tile's
// rows are contiguous in the output.  While a stage's loads are in flight the warp
// already probes the map for the tile after it and issues those loads.  Tiles are
// dealt round-robin over a persistent grid, so neighbouring warps write
// neighbouring pieces of the output at about the same time.
template <int STAGES>
__global__ void __launch_bounds__(kRowThreads)
row_gather_bulk_kernel(const RowJob job) {
  pdl_launch_next();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[kRowWarps][STAGES];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int R = job.rows_per_tile;
  const uint32_t rb = (uint32_t)job.row_bytes;
  const uint32_t stage_bytes = (uint32_t)R * rb;
  unsigned char* wbase = smem_raw + (size_t)warp * STAGES * stage_bytes;
  const int64_t n_tiles = (job.n + R - 1) / R;
  const int64_t stride = (int64_t)gridDim.x * kRowWarps;
  const int64_t slot_mask = ((int64_t)1 << job.owner_shift) - 1;

  if (lane == 0)
    for (int s = 0; s < STAGES; ++s) mbar_init(&s_bar[warp][s], 1);
  mbar_init_fence();
  __syncwarp();
  pdl_wait();

  unsigned vmask[STAGES];  // lanes whose row is being loaded into the stage
  int nrows[STAGES];
  uint32_t parity = 0;     // bit s: phase of stage s to wait for next

  auto issue = [&](int64_t tile, int s) {
    const int64_t first = tile * R;
    const int rows = (int)min((int64_t)R, job.n - first);
    const int64_t id = load_id(job, first, rows, lane);
    char* p = resolve_row(job, first, rows, lane, slot_mask, id);
    const unsigned vm = __ballot_sync(0xffffffffu, p != nullptr);
    if (lane == 0) mbar_arrive_expect_tx(&s_bar[warp][s], (uint32_t)__popc(vm) * rb);
    if (p) bulk_load(wbase + (size_t)s * stage_bytes + (size_t)lane * rb, p, rb, &s_bar[warp][s]);
    vmask[s] = vm;
    nrows[s] = rows;
  };

  // D = STAGES - 1 tiles of loads are in flight while the oldest stage drains its store
  constexpr int D = STAGES - 1;
  int64_t tile = (int64_t)blockIdx.x * kRowWarps + warp;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < D; ++j)
    if (tile + j * stride < n_tiles) issue(tile + j * stride, j);
  while (tile < n_tiles && ok) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      if (tile >= n_tiles || !ok) break;
      const int64_t ahead = tile + D * stride;
      if (ahead < n_tiles) {
        bulk_wait_read<0>();  // the store that last used that stage no longer reads it
        __syncwarp();
        issue(ahead, (s + D) % STAGES);
      }
      // every lane polls: measured faster than one polling lane plus a vote, and fetching
      // the ids a tile ahead of their probe measured slower than loading them here
      if (!mbar_wait_bounded(&s_bar[warp][s], (parity >> s) & 1u)) {
        atomicExch(&g_device_fault, 1);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      parity ^= 1u << s;
      if (ok) {
        unsigned char* buf = wbase + (size_t)s * stage_bytes;
        char* dst = job.flat + tile * R * job.row_bytes;
        const unsigned vm = vmask[s];
        async_proxy_fence();
        if (__popc(vm) == nrows[s]) {
          if (lane == 0 && vm) bulk_store(dst, buf, (uint32_t)nrows[s] * rb);
        } else if ((vm >> lane) & 1u) {
          bulk_store(dst + (size_t)lane * rb, buf + (size_t)lane * rb, rb);
        }
        bulk_commit();
      }
      tile += stride;
    }
  }
  bulk_wait_read<0>();  // shared memory must outlive the stores that read it
}

// The mirror image for set: the tile's update rows are contiguous, so ONE bulk load brings
// them into the stage buffer; each lane then stores its row to where the probe sent it (the
// cached copy on a hit, the host table on a miss) with its own bulk store.
template <int STAGES>
__global__ void __launch_bounds__(kRowThreads)
row_scatter_bulk_kernel(const RowJob job) {
  pdl_launch_next();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[kRowWarps][STAGES];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int R = job.rows_per_tile;
  const uint32_t rb = (uint32_t)job.row_bytes;
  const uint32_t stage_bytes = (uint32_t)R * rb;
  unsigned char* wbase = smem_raw + (size_t)warp * STAGES * stage_bytes;
  const int64_t n_tiles = (job.n + R - 1) / R;
  const int64_t stride = (int64_t)gridDim.x * kRowWarps;
  const int64_t slot_mask = ((int64_t)1 << job.owner_shift) - 1;

  if (lane == 0)
    for (int s = 0; s < STAGES; ++s) mbar_init(&s_bar[warp][s], 1);
  mbar_init_fence();
  __syncwarp();
  pdl_wait();

  char* dst_row[STAGES];  // where this lane's row of the stage goes (nullptr: nowhere)
  uint32_t parity = 0;

  auto issue = [&](int64_t tile, int s) {
    const int64_t first = tile * R;
    const int rows = (int)min((int64_t)R, job.n - first);
    dst_row[s] = resolve_row(job, first, rows, lane, slot_mask, load_id(job, first, rows, lane));
    if (lane == 0) {
      mbar_arrive_expect_tx(&s_bar[warp][s], (uint32_t)rows * rb);
      bulk_load(wbase + (size_t)s * stage_bytes, job.flat + first * job.row_bytes, (uint32_t)rows * rb,
                &s_bar[warp][s]);
    }
  };

  constexpr int D = STAGES - 1;
  int64_t tile = (int64_t)blockIdx.x * kRowWarps + warp;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < D; ++j)
    if (tile + j * stride < n_tiles) issue(tile + j * stride, j);
  while (tile < n_tiles && ok) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      if (tile >= n_tiles || !ok) break;
      const int64_t ahead = tile + D * stride;
      if (ahead < n_tiles) {
        bulk_wait_read<0>();  // every lane's store out of that stage has read it
        __syncwarp();
        issue(ahead, (s + D) % STAGES);
      }
      if (!mbar_wait_bounded(&s_bar[warp][s], (parity >> s) & 1u)) {
        atomicExch(&g_device_fault, 1);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      parity ^= 1u << s;
      if (ok) {
        async_proxy_fence();
        if (dst_row[s])
          bulk_store(dst_row[s], wbase + (size_t)s * stage_bytes + (size_t)lane * rb, rb);
        bulk_commit();
      }
      tile += stride;
    }
  }
  bulk_wait_read<0>();
}

// ---- rows that are not 16-byte units ----------------------------------------------------------
// A row of 602 bytes starts on any even address, and its copy in the output on another one; with
// accesses no wider than both allow, a warp instruction moved 64 bytes.  Here a row travels as the
// 16-byte granules that hold it: one bulk copy per row brings them into a ring buffer like the one
// of row_gather_bulk_kernel, and the warp then writes the tile's output, which is contiguous, in
// aligned 16-byte chunks, each shifted together from two chunks of shared memory (from two rows
// where the chunk holds a seam).  A granule is only read because it holds a byte of the row, so what
// is read beside the row lies in the same 16 bytes, and page, as that byte.

// 16 bytes from byte `sh` (0..15) of the 32 bytes lo | hi
__device__ __forceinline__ uint4 shift_bytes(uint4 lo, uint4 hi, unsigned sh) {
  uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  const bool by2 = sh & 8u, by1 = sh & 4u;
#pragma unroll
  for (int i = 0; i < 6; ++i) w[i] = by2 ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 5; ++i) w[i] = by1 ? w[i + 1] : w[i];
  const unsigned bits = (sh & 3u) * 8u;
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits),
                    __funnelshift_r(w[2], w[3], bits), __funnelshift_r(w[3], w[4], bits));
}

// 16 bytes of shared memory from byte `at` of `base` (16-byte aligned) on
__device__ __forceinline__ uint4 shared_unaligned16(const unsigned char* base, int at) {
  const uint4* a = reinterpret_cast<const uint4*>(base + (at & ~15));
  return shift_bytes(a[0], a[1], (unsigned)at & 15u);
}

// the first `left` bytes of l, the others of r
__device__ __forceinline__ uint4 join_bytes(uint4 l, uint4 r, int left) {
  auto mix = [&](uint32_t x, uint32_t y, int w) {
    const int n = left - 4 * w;  // bytes of this word that belong to l
    const uint32_t keep = n <= 0 ? 0u : (n >= 4 ? 0xFFFFFFFFu : (1u << (8 * n)) - 1u);
    return (x & keep) | (y & ~keep);
  };
  return make_uint4(mix(l.x, r.x, 0), mix(l.y, r.y, 1), mix(l.z, r.z, 2), mix(l.w, r.w, 3));
}

// bytes [from, to) of v to dst + from .. (a chunk whose other bytes are not this tile's to write)
__device__ __forceinline__ void store_bytes(char* dst, uint4 v, int from, int to) {
  for (int i = from; i < to; ++i) {
    const uint32_t w = i < 8 ? (i < 4 ? v.x : v.y) : (i < 12 ? v.z : v.w);
    dst[i] = (char)(w >> (8 * (i & 3)));
  }
}

// Shared memory between two rows of a stage buffer: the granules of a row that starts on any byte.
__host__ __device__ constexpr int64_t ragged_pitch(int64_t row_bytes) { return (row_bytes + 30) & ~(int64_t)15; }
constexpr int kRaggedPad = 32;  // in front of and behind a warp's buffers: what seams read past a row is never used

template <int STAGES>
__global__ void __launch_bounds__(kRowThreads)
row_gather_ragged_kernel(const RowJob job) {
  pdl_launch_next();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_bar[kRowWarps][STAGES];
  const unsigned full = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int R = job.rows_per_tile;
  const int rb = (int)job.row_bytes, pitch = (int)ragged_pitch(job.row_bytes);
  const int stage_bytes = R * pitch;
  unsigned char* wbase = smem_raw + (size_t)warp * (STAGES * stage_bytes + 2 * kRaggedPad) + kRaggedPad;
  const int64_t n_tiles = (job.n + R - 1) / R;
  const int64_t stride = (int64_t)gridDim.x * kRowWarps;
  const int64_t slot_mask = ((int64_t)1 << job.owner_shift) - 1;
  const int step_row = 512 / rb, step_off = 512 % rb;

  if (lane == 0)
    for (int s = 0; s < STAGES; ++s) mbar_init(&s_bar[warp][s], 1);
  mbar_init_fence();
  __syncwarp();
  pdl_wait();

  unsigned vmask[STAGES];  // lanes whose row is being loaded into the stage
  int start[STAGES];       // byte of this lane's slot at which its row starts
  uint32_t parity = 0;     // bit s: phase of stage s to wait for next

  int64_t tile = (int64_t)blockIdx.x * kRowWarps + warp;
  if (tile >= n_tiles) return;
  RowCursor cursor(job, tile, stride, slot_mask);
  int64_t issued = 0;  // tiles of this warp
  auto issue = [&](int s) {
    const char* p = cursor.row_of(job, issued++, slot_mask);
    const int sh = (int)((uintptr_t)p & 15);
    const uint32_t bytes = p ? (uint32_t)(sh + rb + 15) & ~15u : 0u;
    const uint32_t total = __reduce_add_sync(full, bytes);
    if (lane == 0) mbar_arrive_expect_tx(&s_bar[warp][s], total);
    __syncwarp();
    if (p) bulk_load(wbase + s * stage_bytes + (int)lane * pitch, p - sh, bytes, &s_bar[warp][s]);
    vmask[s] = __ballot_sync(full, p != nullptr);
    start[s] = sh;
  };

  constexpr int D = STAGES - 1;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < D; ++j)
    if (tile + j * stride < n_tiles) issue(j);
  while (tile < n_tiles && ok) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      if (tile >= n_tiles || !ok) break;
      const int64_t ahead = tile + D * stride;
      __syncwarp();  // every lane has read what the buffer filled next held
      if (ahead < n_tiles) issue((s + D) % STAGES);
      if (!mbar_wait_bounded(&s_bar[warp][s], (parity >> s) & 1u)) {
        atomicExch(&g_device_fault, 1);
        ok = false;
      }
      ok = __all_sync(full, ok);
      parity ^= 1u << s;
      if (ok) {
        const unsigned char* buf = wbase + s * stage_bytes;
        const unsigned vm = vmask[s];
        const int rows = (int)min((int64_t)R, job.n - tile * R);
        char* out = job.flat + tile * R * job.row_bytes;
        const int d = (int)((uintptr_t)out & 15);  // the tile starts at byte d of its first chunk
        char* chunk0 = out - d;
        const int n_chunks = (rows * rb + d + 15) >> 4;
        // ---- chunks inside one row; the lane's starts at byte `off` of row `row`
        int row = 0, off = (int)lane * 16 - d;
        if (off < 0) {  // the tile's first chunk is a seam
          row = -1;
          off += rb;
        } else if (off >= rb) {  // off <= 496, and no row is shorter than 256
          row = 1;
          off -= rb;
        }
        for (int c0 = 0; c0 < n_chunks; c0 += 32) {
          const int at = __shfl_sync(full, start[s], row & 31) + off;
          if (off + 16 <= rb && row < rows && row >= 0 && (vm >> row & 1u))
            st_stream16(chunk0 + (c0 + (int)lane) * 16, shared_unaligned16(buf, row * pitch + at));
          off += step_off;
          row += step_row;
          if (off >= rb) {
            off -= rb;
            ++row;
          }
        }
        // ---- seams, one per lane: the chunk that holds the start of row b (b = rows: the tile's end)
        for (int b0 = 0; b0 <= rows; b0 += 32) {
          const int b = b0 + (int)lane;
          const int at0 = __shfl_sync(full, start[s], (b - 1) & 31), at1 = __shfl_sync(full, start[s], b & 31);
          const int left = (b * rb + d) & 15;  // bytes of the chunk in front of the seam
          if (b > rows || left == 0) continue;
          const bool has0 = b > 0 && (vm >> (b - 1) & 1u), has1 = b < rows && (vm >> b & 1u);
          uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
          if (has0) v0 = shared_unaligned16(buf, (b - 1) * pitch + at0 + rb - left);
          if (has1) v1 = shared_unaligned16(buf, b * pitch + at1 - left);
          const uint4 v = join_bytes(v0, v1, left);
          char* dst = out + b * rb - left;
          if (has0 && has1)
            st_stream16(dst, v);
          else
            store_bytes(dst, v, has0 ? 0 : left, has1 ? 16 : (has0 ? left : 0));
        }
      }
      tile += stride;
    }
  }
}

// SET == false: table row -> flat (fetch).  SET == true: flat -> table row.
template <int VEC, bool SET, int U>
__global__ void __launch_bounds__(kRowThreads) row_copy_kernel(const RowJob job) {
  pdl_prologue();
  using V = typename VecT<VEC>::type;
  __shared__ char* s_row[kRowWarps][32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int R = job.rows_per_tile;
  const int64_t n_tiles = (job.n + R - 1) / R;
  const uint32_t cpr = (uint32_t)(job.row_bytes / VEC);  // chunks per row
  const uint32_t step_row = 32u / cpr, step_off = 32u % cpr;
  const int64_t slot_mask = ((int64_t)1 << job.owner_shift) - 1;

  for (int64_t tile = (int64_t)blockIdx.x * kRowWarps + warp; tile < n_tiles;
       tile += (int64_t)gridDim.x * kRowWarps) {
    const int64_t first = tile * R;
    const int rows = (int)min((int64_t)R, job.n - first);

    // ---- phase A: one request per lane -> row address
    {
      char* p = resolve_row(job, first, rows, lane, slot_mask, load_id(job, first, rows, lane));
      __syncwarp();  // previous tile's readers are done with s_row
      s_row[warp][lane] = p;
      __syncwarp();
    }

    // ---- phase B: flat chunk copy
    const uint32_t total = (uint32_t)rows * cpr;
    char* flat = job.flat + first * job.row_bytes;
    uint32_t row = lane / cpr, off = lane % cpr;
    for (uint32_t c0 = 0; c0 < total; c0 += 32u * U) {
      V v[U];
      char* tp[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t c = c0 + u * 32u + lane;
        tp[u] = nullptr;
        if (c < total) {
          char* base = s_row[warp][row];
          if (base) tp[u] = base + (size_t)off * VEC;
        }
        if (tp[u]) v[u] = load_chunk<VEC>(SET ? flat + (size_t)c * VEC : tp[u]);
        off += step_off;
        row += step_row;
        if (off >= cpr) {
          off -= cpr;
          ++row;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t c = c0 + u * 32u + lane;
        if (tp[u]) store_chunk<VEC>(SET ? tp[u] : flat + (size_t)c * VEC, v[u]);
      }
    }
  }
}

// Fused insert/overwrite: probe-or-claim the key, then write the row to the
// slot the map now holds for it.  (80 registers, 3 CTAs per SM: forcing 4 CTAs with 64
// registers measured 4 % slower on 4,000,000 keys x 512 bytes.)
template <int VEC, int U>
__global__ void __launch_bounds__(kRowThreads)
insert_set_kernel(MapView map, char* gpu_base, const void* keys, int keys64, const void* slots,
                  int slots64, int64_t n, int64_t row_bytes, const char* update, int R,
                  int64_t* meta) {
  using V = typename VecT<VEC>::type;
  __shared__ char* s_row[kRowWarps][32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n_tiles = (n + R - 1) / R;
  const uint32_t cpr = (uint32_t)(row_bytes / VEC);
  const uint32_t step_row = 32u / cpr, step_off = 32u % cpr;
  int64_t total_new = 0;

  for (int64_t tile = (int64_t)blockIdx.x * kRowWarps + warp; tile < n_tiles;
       tile += (int64_t)gridDim.x * kRowWarps) {
    const int64_t first = tile * R;
    const int rows = (int)min((int64_t)R, n - first);
    {
      const bool valid = (int)lane < rows;
      const int64_t k = valid ? load_int(keys, keys64, first + lane) : kEmptyKey;
      const int64_t want = valid ? load_int(slots, slots64, first + lane) : -1;
      int n_new = 0;
      const int64_t got = warp_insert(map, k, want, valid, /*assign=*/false, meta, &n_new);
      total_new += n_new;
      __syncwarp();
      s_row[warp][lane] = (valid && got >= 0) ? gpu_base + got * row_bytes : nullptr;
      __syncwarp();
    }
    const uint32_t total = (uint32_t)rows * cpr;
    const char* flat = update + first * row_bytes;
    uint32_t row = lane / cpr, off = lane % cpr;
    for (uint32_t c0 = 0; c0 < total; c0 += 32u * U) {
      V v[U];
      char* tp[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t c = c0 + u * 32u + lane;
        tp[u] = nullptr;
        if (c < total) {
          char* base = s_row[warp][row];
          if (base) tp[u] = base + (size_t)off * VEC;
        }
        if (tp[u]) v[u] = load_chunk<VEC>(flat + (size_t)c * VEC);
        off += step_off;
        row += step_row;
        if (off >= cpr) {
          off -= cpr;
          ++row;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (tp[u]) store_chunk<VEC>(tp[u], v[u]);
    }
  }
  if (lane == 0 && total_new)
    atomicAdd(reinterpret_cast<unsigned long long*>(meta + 1), (unsigned long long)total_new);
}

// ---- host side ---------------------------------------------------------------

static int pick_vec(int64_t row_bytes, std::initializer_list<const void*> ptrs) {
  uintptr_t bits = (uintptr_t)row_bytes;
  for (const void* p : ptrs) bits |= (uintptr_t)p;
  if ((bits & 15) == 0) return 16;
  if ((bits & 7) == 0) return 8;
  if ((bits & 3) == 0) return 4;
  if ((bits & 1) == 0) return 2;
  return 1;
}

// Rows per warp tile: 32 when there is enough work to fill the GPU, fewer for
// small batches so that they still spread over all SMs.
static int pick_rows_per_tile(int64_t n) {
  const int64_t warps_wanted = (int64_t)sm_count() * 32;
  int r = 32;
  while (r > 1 && (n + r - 1) / r < warps_wanted) r >>= 1;
  return r;
}

// Persistent grid: never more CTAs than are resident at once (tiles are dealt round-robin
// inside the kernels), so there is no partly filled last wave.  The occupancy of a kernel with so
// much shared memory is asked for once per device (1 us, a fifth of a small call) and kept beside the kernel.
template <typename Kernel>
static unsigned grid_for_tiles(Kernel kernel, KeptOccupancy* kept, int dev, int64_t n, int R, size_t smem = 0) {
  const int64_t tiles = (n + R - 1) / R;
  int64_t blocks = (tiles + kRowWarps - 1) / kRowWarps;
  const int occ = kept->get(dev, smem, [&](int* ctas) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, kernel, kRowThreads, smem) == cudaSuccess;
  });
  const int64_t resident = (int64_t)sm_count() * occ;
  if (blocks > resident) blocks = resident;
  return (unsigned)(blocks < 1 ? 1 : blocks);
}

template <int VEC, bool SET>
static int launch_lsu(const RowJob& job, cudaStream_t s) {
  static KeptOccupancy kept;
  int dev = 0;
  SHMT_CUDA_TRY(cudaGetDevice(&dev));
  const unsigned grid = grid_for_tiles(row_copy_kernel<VEC, SET, 8>, &kept, dev, job.n, job.rows_per_tile);
  SHMT_CUDA_TRY(launch_kernel(true, row_copy_kernel<VEC, SET, 8>, grid, kRowThreads, 0, s, job));
  return SHMT_OK;
}

// Ring geometry of the bulk path: two buffers per warp of about 2 KB each (5 rows of
// 400 bytes): measured best on B200 among 0.5 .. 12 KB buffers and 2 .. 4 stages.
constexpr int kBulkStages = 2;
constexpr int64_t kBulkStageBytes = 2048;
// A fetch looks a tile's rows up in one go and waits for it, so few rows a tile means few lookups on their way.
// Rows of 512 bytes and more therefore come 6 a buffer, as long as these fit.  60,000 rows by popularity / drawn evenly
// from 1.6 GB: 512 bytes 14.4 -> 11.9 us / 18.1 -> 14.9, 800 20.7 -> 16.9 / 24.6 -> 22.4, 1,200 34 -> 20.4 / 37.0 -> 29.8.
// An output much smaller than the L2 cache stays there.  A larger one is written to HBM while rows are read, and rows drawn
// evenly come from HBM too: then six rows of 512 to 930 bytes are slower (512 bytes, six and four rows: 90 MB 38.1 us and 38.8, 120 MB
// 50.4 and 48.6, 600 MB 236 and 224; 640: 37.1 and 38.3, 48.5 and 47.5, 234 and 212; 896: 35.2 and 37.3, 47.4 and 47.2, 227
// and 208; from 960 on: 230 and 233, 1,008 233 and 240, 1,200 222 and 255), and so are six of 1,550 to 1,730 (1,664: 210, one row 203,
// five 196).  By popularity six are faster (512: 600 MB 137 and 167; 1,664: 142, five 148), but whether a call's rows
// repeat is not known here, and a frontier's are distinct.
// Sets have their own line: 512 bytes 124 us with 4 rows and 129 with 6, 800 bytes 189 with 2 and 208.
constexpr int64_t kWideRowBytes = 512, kWideStageBytes = 12800;
constexpr int kWideRows = 6;
constexpr int64_t kLargeOutBytes = (int64_t)88 << 20, kLargeOutWideRowBytes = 960, kLargeOutFewRowBytes[2] = {1536, 1760};
constexpr int kLargeOutFewRows = 5;
constexpr size_t kBulkSmemMax = 200 * 1024;

// Rows per ring buffer, 0 if the rows are not 16-byte units or do not fit.
static int bulk_rows_per_stage(int64_t n, int64_t row_bytes, int vec, int R_small, bool set) {
  if (vec != 16) return 0;
  static const int forced = [] {
    const char* e = getenv("SHMT_BULK_ROWS");
    return e ? atoi(e) : 0;
  }();
  int64_t r = forced > 0 ? forced : kBulkStageBytes / row_bytes;
  const bool large = n > kLargeOutBytes / row_bytes;
  if (forced <= 0 && !set && row_bytes >= (large ? kLargeOutWideRowBytes : kWideRowBytes)) {
    const bool few = large && row_bytes > kLargeOutFewRowBytes[0] && row_bytes < kLargeOutFewRowBytes[1];
    const int most = few ? kLargeOutFewRows : kWideRows;
    r = kWideStageBytes / row_bytes;
    if (r > most) r = most;
  }
  if (r < 1) r = 1;
  if (r > 32) r = 32;
  if (r > R_small) r = R_small;
  if ((size_t)kRowWarps * kBulkStages * r * row_bytes > kBulkSmemMax) return 0;
  return (int)r;
}

template <bool SET>
static int launch_bulk(RowJob job, int R, cudaStream_t s) {
  auto kernel = SET ? row_scatter_bulk_kernel<kBulkStages> : row_gather_bulk_kernel<kBulkStages>;
  static bool configured[64] = {false};
  int dev = 0;
  SHMT_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && !configured[dev]) {
    SHMT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kBulkSmemMax));
    configured[dev] = true;
  }
  job.rows_per_tile = R;
  const size_t smem = (size_t)kRowWarps * kBulkStages * R * job.row_bytes;
  static KeptOccupancy kept;
  const unsigned blocks = grid_for_tiles(kernel, &kept, dev, job.n, R, smem);
  SHMT_CUDA_TRY(launch_kernel(true, kernel, blocks, kRowThreads, smem, s, job));
  return SHMT_OK;
}

// Rows that are not 16-byte units.  Buffers of about 5 KB per warp (150,001 rows of 602 bytes: 3.4
// TB/s read + written with 2 KB, 4.3 with 3 KB, 4.8 with 4 KB, 5.0 with 5 KB; a third buffer gave
// nothing).  The line at 256 bytes: there the narrow copy of row_copy_kernel still has 2.3 (4-byte
// rows: 3.4) against 4.2 TB/s and 26 (33) against 35 GB/s from a host table, below it the seams and
// granules read at both ends of a row outweigh the wider access (132 bytes: 2.9 against 2.3 TB/s, 28
// against 24 GB/s).  Rows of 8-byte units have a faster narrow copy, which is level at 408 bytes
// (4.8 against 5.0 TB/s, 41.0 against 40.9 GB/s) and behind at 600 (4.2 against 5.1, 43.1 against 44.2).
// A small batch read from the host alone is a wait for its few rows, to which granules add a trip through
// shared memory: rows of 4- and 8-byte units take the narrow copy up to 512 KB a batch, and up to 4 MB where
// they are shorter than 512 and 600 bytes (300 rows of 808 bytes 9.3 us against 9.9, 3,000 of 260 bytes 24.0
// against 26.7, of 520 38.5 against 40.0; but 20,000 of 260 bytes 158 against 146, of 520 245 against 237).
// 2-byte units are faster in granules from 1,000 rows of 258 bytes on (12.6 against 11.7).
// A batch that may hit the cache takes granules whatever its size: how many of its rows miss is not known here.
// Where all hit, the narrow copy is 0.5 to 3 us faster up to about 40 MB of 8-byte units or 5 MB of 4-byte units
// (30,000 rows of 1,000 bytes 11.3 against 12.4); where a fifth of those rows miss, granules are by 5 (135
// against 130).
constexpr int kRaggedStages = 2;
constexpr int64_t kRaggedStageBytes = 5120;
constexpr int64_t kRaggedMinBytes = 256, kRaggedMinBytes8 = 512;
constexpr int64_t kRaggedHostBytes = 512 << 10, kRaggedHostBytesShort = 4 << 20;  // of a batch from the host alone
constexpr int64_t kRaggedHostRow4 = 512, kRaggedHostRow8 = 600;                     // rows below are short

static size_t ragged_smem_bytes(int64_t row_bytes, int R) {
  return (size_t)kRowWarps * ((size_t)kRaggedStages * R * ragged_pitch(row_bytes) + 2 * kRaggedPad);
}

// Rows per ring buffer, 0 if the batch is not to gain or its rows do not fit.
static int ragged_rows_per_stage(const RowJob& job, int vec) {
  const int64_t row_bytes = job.row_bytes;
  if (vec == 16 || row_bytes < (vec == 8 ? kRaggedMinBytes8 : kRaggedMinBytes)) return 0;
  if (job.mode == MODE_HOST && vec >= 4) {
    const bool is_short = row_bytes < (vec == 8 ? kRaggedHostRow8 : kRaggedHostRow4);
    if (job.n * row_bytes < (is_short ? kRaggedHostBytesShort : kRaggedHostBytes)) return 0;
  }
  int64_t r = kRaggedStageBytes / ragged_pitch(row_bytes);
  if (r < 1) r = 1;
  if (r > 32) r = 32;
  if (r > job.rows_per_tile) r = job.rows_per_tile;
  return ragged_smem_bytes(row_bytes, (int)r) > kBulkSmemMax ? 0 : (int)r;
}

static int launch_ragged(RowJob job, int R, cudaStream_t s) {
  auto kernel = row_gather_ragged_kernel<kRaggedStages>;
  static bool configured[64] = {false};
  int dev = 0;
  SHMT_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 64 && !configured[dev]) {
    SHMT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBulkSmemMax));
    configured[dev] = true;
  }
  job.rows_per_tile = R;
  const size_t smem = ragged_smem_bytes(job.row_bytes, R);
  static KeptOccupancy kept;
  SHMT_CUDA_TRY(launch_kernel(true, kernel, grid_for_tiles(kernel, &kept, dev, job.n, R, smem), kRowThreads, smem, s, job));
  return SHMT_OK;
}

template <bool SET>
static int launch_row_copy(const RowJob& job, int vec, cudaStream_t s) {
  {
    static const bool no_bulk = getenv("SHMT_NO_BULK") != nullptr;
    const int R = no_bulk ? 0 : bulk_rows_per_stage(job.n, job.row_bytes, vec, job.rows_per_tile, SET);
    if (R >= 1) return launch_bulk<SET>(job, R, s);
    const int ragged = SET || no_bulk ? 0 : ragged_rows_per_stage(job, vec);
    if (ragged >= 1) return launch_ragged(job, ragged, s);
  }
  switch (vec) {
    case 16: return launch_lsu<16, SET>(job, s);
    case 8: return launch_lsu<8, SET>(job, s);
    case 4: return launch_lsu<4, SET>(job, s);
    case 2: return launch_lsu<2, SET>(job, s);
    default: return launch_lsu<1, SET>(job, s);
  }
}

static int check_common(const char* who, const void* idx, int idx_dtype, int64_t n,
                        int64_t row_bytes) {
  SHMT_REQUIRE(valid_int_dtype(idx_dtype), "%s: indices can only be int32 or int64", who);
  SHMT_REQUIRE(n >= 0, "%s: negative count", who);
  SHMT_REQUIRE(row_bytes > 0 && row_bytes < ((int64_t)1 << 26),
               "%s: row_bytes %lld out of range (1 .. 64 MiB)", who, (long long)row_bytes);
  SHMT_REQUIRE(n == 0 || idx != nullptr, "%s: indices are null", who);
  return SHMT_OK;
}

static int fill_mode(const char* who, RowJob& job, const shmt_map* map, const void* mask,
                     int mask_dtype) {
  job.map = view_of(map);
  job.mask = mask;
  job.mask64 = mask_dtype == SHMT_I64;
  if (map) {
    SHMT_REQUIRE(mask == nullptr, "%s: give a map or a mask, not both", who);
    job.mode = MODE_MAP;
  } else if (mask) {
    SHMT_REQUIRE(valid_int_dtype(mask_dtype), "%s: mask can only be int32 or int64", who);
    job.mode = MODE_MASK;
  } else {
    job.mode = MODE_HOST;
  }
  return SHMT_OK;
}

}  // namespace shmt

using namespace shmt;

extern "C" {

int shmt_device_fault(int* out_code) {
  SHMT_REQUIRE(out_code != nullptr, "shmt_device_fault: out_code is null");
  int code = 0, zero = 0;
  SHMT_CUDA_TRY(cudaMemcpyFromSymbol(&code, g_device_fault, sizeof(int)));
  if (code) SHMT_CUDA_TRY(cudaMemcpyToSymbol(g_device_fault, &zero, sizeof(int)));
  *out_code = code;
  return SHMT_OK;
}

int shmt_fetch(const shmt_map* map, const void* mask, int mask_dtype, const void* host_base,
               const void* gpu_base, const void* idx, int idx_dtype, int64_t n, int64_t row_bytes,
               void* out, void* stream) {
  if (int rc = check_common("shmt_fetch", idx, idx_dtype, n, row_bytes)) return rc;
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(out != nullptr, "shmt_fetch: out is null");
  DeviceGuard guard(map ? map->device : device_of_pointer(out));
  RowJob job{};
  if (int rc = fill_mode("shmt_fetch", job, map, mask, mask_dtype)) return rc;
  SHMT_REQUIRE(job.mode == MODE_HOST ? host_base != nullptr : (gpu_base || host_base),
               "shmt_fetch: the table pointer this mode reads is null");
  job.host = static_cast<char*>(const_cast<void*>(host_base));
  job.bases[0] = static_cast<char*>(const_cast<void*>(gpu_base));
  job.owner_shift = 62;
  job.idx = idx;
  job.idx64 = idx_dtype == SHMT_I64;
  job.n = n;
  job.row_bytes = row_bytes;
  job.flat = static_cast<char*>(out);
  job.rows_per_tile = pick_rows_per_tile(n);
  const int vec = pick_vec(row_bytes, {host_base, gpu_base, out});
  return launch_row_copy<false>(job, vec, static_cast<cudaStream_t>(stream));
}

int shmt_fetch_partitioned(const shmt_map* map, const void* const* bases, int n_bases,
                           int owner_shift, const void* host_base, const void* idx, int idx_dtype,
                           int64_t n, int64_t row_bytes, void* out, void* stream) {
  if (int rc = check_common("shmt_fetch_partitioned", idx, idx_dtype, n, row_bytes)) return rc;
  SHMT_REQUIRE(map != nullptr, "shmt_fetch_partitioned: map is null");
  SHMT_REQUIRE(bases != nullptr && n_bases >= 1 && n_bases <= kMaxBases,
               "shmt_fetch_partitioned: 1..%d row buffers", kMaxBases);
  SHMT_REQUIRE(owner_shift >= 1 && owner_shift <= 62, "shmt_fetch_partitioned: owner_shift 1..62");
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(out != nullptr, "shmt_fetch_partitioned: out is null");
  DeviceGuard guard(map->device);
  RowJob job{};
  job.map = view_of(map);
  job.mode = MODE_MAP;
  job.host = static_cast<char*>(const_cast<void*>(host_base));
  uintptr_t align = 0;
  for (int g = 0; g < n_bases; ++g) {
    SHMT_REQUIRE(bases[g] != nullptr, "shmt_fetch_partitioned: row buffer %d is null", g);
    job.bases[g] = static_cast<char*>(const_cast<void*>(bases[g]));
    align |= (uintptr_t)bases[g];
  }
  // a value naming an owner beyond n_bases reads bases[0]; owners are the caller's contract
  for (int g = n_bases; g < kMaxBases; ++g) job.bases[g] = job.bases[0];
  job.owner_shift = owner_shift;
  job.idx = idx;
  job.idx64 = idx_dtype == SHMT_I64;
  job.n = n;
  job.row_bytes = row_bytes;
  job.flat = static_cast<char*>(out);
  job.rows_per_tile = pick_rows_per_tile(n);
  const int vec = pick_vec(row_bytes, {host_base, (const void*)align, out});
  return launch_row_copy<false>(job, vec, static_cast<cudaStream_t>(stream));
}

int shmt_set(const shmt_map* map, const void* mask, int mask_dtype, void* host_base,
             void* gpu_base, const void* idx, int idx_dtype, int64_t n, int64_t row_bytes,
             const void* update, void* stream) {
  if (int rc = check_common("shmt_set", idx, idx_dtype, n, row_bytes)) return rc;
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(update != nullptr, "shmt_set: update is null");
  DeviceGuard guard(map ? map->device : device_of_pointer(update));
  RowJob job{};
  if (int rc = fill_mode("shmt_set", job, map, mask, mask_dtype)) return rc;
  SHMT_REQUIRE(job.mode == MODE_HOST ? host_base != nullptr : (gpu_base || host_base),
               "shmt_set: the table pointer this mode writes is null");
  job.host = static_cast<char*>(host_base);
  job.bases[0] = static_cast<char*>(gpu_base);
  job.owner_shift = 62;
  job.idx = idx;
  job.idx64 = idx_dtype == SHMT_I64;
  job.n = n;
  job.row_bytes = row_bytes;
  job.flat = static_cast<char*>(const_cast<void*>(update));
  job.rows_per_tile = pick_rows_per_tile(n);
  const int vec = pick_vec(row_bytes, {host_base, gpu_base, update});
  return launch_row_copy<true>(job, vec, static_cast<cudaStream_t>(stream));
}

int shmt_insert_set(shmt_map* map, void* gpu_base, const void* keys, int key_dtype,
                    const void* slots, int slots_dtype, int64_t n, int64_t row_bytes,
                    const void* update, void* stream) {
  if (int rc = check_common("shmt_insert_set", keys, key_dtype, n, row_bytes)) return rc;
  SHMT_REQUIRE(map != nullptr, "shmt_insert_set: map is null");
  SHMT_REQUIRE(valid_int_dtype(slots_dtype), "shmt_insert_set: slots can only be int32 or int64");
  if (n == 0) return SHMT_OK;
  SHMT_REQUIRE(gpu_base && slots && update, "shmt_insert_set: gpu_base/slots/update are null");
  DeviceGuard guard(map->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int R = pick_rows_per_tile(n);
  static KeptOccupancy kept;
  const unsigned grid = grid_for_tiles(insert_set_kernel<16, 8>, &kept, map->device, n, R);
  const int vec = pick_vec(row_bytes, {gpu_base, update});
  char* g = static_cast<char*>(gpu_base);
  const char* u = static_cast<const char*>(update);
  const int k64 = key_dtype == SHMT_I64, s64 = slots_dtype == SHMT_I64;
  // the status word reports on this call only (see shmt_map_insert)
  SHMT_CUDA_TRY(cudaMemsetAsync(map->d_meta, 0, sizeof(int64_t), s));
  switch (vec) {
    case 16: insert_set_kernel<16, 8><<<grid, kRowThreads, 0, s>>>(map->view, g, keys, k64, slots, s64, n, row_bytes, u, R, map->d_meta); break;
    case 8: insert_set_kernel<8, 8><<<grid, kRowThreads, 0, s>>>(map->view, g, keys, k64, slots, s64, n, row_bytes, u, R, map->d_meta); break;
    case 4: insert_set_kernel<4, 8><<<grid, kRowThreads, 0, s>>>(map->view, g, keys, k64, slots, s64, n, row_bytes, u, R, map->d_meta); break;
    case 2: insert_set_kernel<2, 8><<<grid, kRowThreads, 0, s>>>(map->view, g, keys, k64, slots, s64, n, row_bytes, u, R, map->d_meta); break;
    default: insert_set_kernel<1, 8><<<grid, kRowThreads, 0, s>>>(map->view, g, keys, k64, slots, s64, n, row_bytes, u, R, map->d_meta); break;
  }
  SHMT_CUDA_TRY(cudaGetLastError());
  int64_t meta[2] = {0, 0};
  SHMT_CUDA_TRY(cudaMemcpyAsync(meta, map->d_meta, sizeof(meta), cudaMemcpyDeviceToHost, s));
  SHMT_CUDA_TRY(cudaStreamSynchronize(s));
  map->size = meta[1];
  if (meta[0] == DEV_OVERFLOW) {
    set_error("shmt_insert_set: table overflow (%lld keys stored, capacity %lld)",
              (long long)meta[1], (long long)map->capacity);
    return SHMT_ERR_CAPACITY;
  }
  return SHMT_OK;
}

}  // extern "C"
