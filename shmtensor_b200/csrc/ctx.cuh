// Per-device context: reusable scratch + result words (host side).
#pragma once

#include "common.cuh"

namespace shmt {

// Result words handed to the host without a copy and before the stream drains: the thread that
// completes them stores them into the context's pinned host words and then a sequence number,
// which the host polls for.  Whatever the stream still runs behind that point must not produce
// results or errors the host needs.
//
// A note (n_words = 0) is two numbers, stored to host[flag_at] and the word behind it by the thread that has
// them, as soon as it has them and in no order with anything; the host has set both words to -1.
struct HostPost {
  int64_t* host;         // pinned host words as the device sees them; nullptr = no post
  const int64_t* words;  // device words to mirror
  int n_words;
  int flag_at;           // index of the sequence word (the last pinned word)
  int64_t seq;           // stored to host[flag_at] after the words
  int64_t* done;         // zeroed device word counting the CTAs that have finished
};

}  // namespace shmt

struct shmt_ctx {
  int device = 0;
  char* scratch = nullptr;      // device scratch, grown geometrically; the first
  size_t scratch_bytes = 0;     // 256 bytes are the result words (status, result, ticket ...)
  int64_t* h_words = nullptr;   // pinned host mirror of the result words
  // Relabel table (16-byte slots, see relabel.cuh), empty between calls: the kernels that number the
  // ids empty every slot they leave, so no per-call memset is needed.
  char* table = nullptr;
  size_t table_bytes = 0;
  bool table_dirty = false;     // a failed call may have left entries behind
  // Words of mini-batches (RelTable in relabel.cuh), in a block of their own: they hold numbers from words_tag on,
  // which would be taken for slots, and a table that grew for them would leave captured relabels without theirs.
  unsigned* words = nullptr;
  size_t words_bytes = 0;
  unsigned words_tag = 0;
  bool words_dirty = false;     // a failed call may have left numbers below words_tag behind
  bool words_reserved = false;  // the caller sized the context for mini-batches: none of them grows it for words
  // Early hand-over of result words (see HostPost): sequence number of the last post, and an
  // event behind the kernels that were still running when the call returned.
  int64_t post_seq = 0;
  cudaEvent_t tail_event = nullptr;
  unsigned long long tail_stream = 0;  // its id: a handle may be another stream's by now
  bool tail_pending = false;
  // The mini-batch that has been queued and not yet been waited for (shmt_minibatch_start).
  struct {
    shmt::HostPost post{};
    void* stream = nullptr;
    int n_hops = 0;  // 0: none
    int64_t n_seeds = 0;
    bool noted = false;  // sizes of all hops but the last come as notes
  } batch;
  // Ticket, count of finished CTAs and tile descriptors of small scans: zero between calls, put back by
  // the scan kernel itself (see scan.cu).
  char* scan_state = nullptr;
  int64_t* scan_words() const { return reinterpret_cast<int64_t*>(scan_state); }
  int64_t* d_words() const { return reinterpret_cast<int64_t*>(scratch); }
  char* region() const { return scratch + 256; }
};

namespace shmt {

constexpr int kCtxWords = 128;
constexpr int kNoteWord = 96;  // notes of a mini-batch's hops in shmt_ctx::h_words, two words each
constexpr int kSmallScanTiles = 512;  // tiles whose descriptors live in shmt_ctx::scan_state
constexpr size_t kScanStateBytes = 16 + (size_t)kSmallScanTiles * 16;
enum : int { W_STATUS = 0, W_RESULT = 1, W_TICKET = 2, W_DONE = 3 };

// Make sure ctx->region() holds at least `bytes` (256-byte aligned base).
int ctx_reserve(shmt_ctx* ctx, size_t bytes, cudaStream_t stream);

// Make sure ctx->table holds at least `bytes`, empty (all ones to begin with).  This and the next one are for callers that
// have been through ctx_reserve, which waits for the context's use in another stream.
int ctx_reserve_table(shmt_ctx* ctx, size_t bytes, cudaStream_t stream);

// Make sure ctx->words holds at least `bytes`, every word of them above words_tag - 1.
int ctx_reserve_words(shmt_ctx* ctx, size_t bytes, cudaStream_t stream);

// A failed call may have left entries in the table and the words.
inline void ctx_table_failed(shmt_ctx* ctx) { ctx->table_dirty = ctx->words_dirty = true; }

// `count` numbers below all that the words hold: *first and those behind it.
int ctx_take_tags(shmt_ctx* ctx, unsigned count, unsigned* first, cudaStream_t stream);

// Copy the first `n_words` result words to the host and wait for `stream`.
// Returns SHMT_ERR_TIMEOUT / SHMT_ERR_CAPACITY if the kernel flagged either.
int ctx_fetch_words(shmt_ctx* ctx, cudaStream_t stream, const char* what);
// The same check on words that are already in ctx->h_words.
int ctx_status_of_words(shmt_ctx* ctx, const char* what);

#ifdef __CUDACC__
// Called by a whole warp: a word per lane.  One thread copying word by word took 0.6 us for each (the
// next load waits behind the store of the one before), 17 us for the sizes of a three-hop mini-batch,
// all of it on the way to the host.  The words are final for every lane (behind a barrier, or a fence
// and a __syncwarp).  The sequence number is a release at system scope by one lane, behind a
// __syncwarp: it carries the words of all lanes to the host.
__device__ __forceinline__ void post_to_host(const HostPost& p) {
  if (!p.host) return;
  const unsigned lane = threadIdx.x & 31;
  for (int i = (int)lane; i < p.n_words; i += 32)
    *reinterpret_cast<volatile int64_t*>(p.host + i) = ld_relaxed64(p.words + i);
  __syncwarp();
  if (lane == 0) st_release_sys64(p.host + p.flag_at, p.seq);
}

// The same with the first four words, as far as they are not W_RESULT, zero, and by a warp that has the result.
__device__ __forceinline__ void post_result(const HostPost& p, int64_t result) {
  if (!p.host) return;
  const int lane = (int)(threadIdx.x & 31);
  if (lane < p.n_words) *reinterpret_cast<volatile int64_t*>(p.host + lane) = lane == W_RESULT ? result : 0;
  __syncwarp();
  if (lane == 0) st_release_sys64(p.host + p.flag_at, p.seq);
}

__device__ __forceinline__ void post_note(const HostPost& p, int64_t a, int64_t b) {
  *reinterpret_cast<volatile int64_t*>(p.host + p.flag_at) = a;
  *reinterpret_cast<volatile int64_t*>(p.host + p.flag_at + 1) = b;
}

// True on every lane of the calling warp if its CTA is the last of `n_ctas` to count itself out at `done`
// (zero when the kernel starts).  What the other CTAs did before they counted themselves out, as far
// as their calling warp had seen it (a CTA-wide barrier before the call), has then happened for every lane:
// fences around one lane's atomic, and a __syncwarp, for a shuffle orders no memory.
__device__ __forceinline__ bool last_to_finish(int64_t* done, int64_t n_ctas) {
  unsigned long long before = 0;
  if ((threadIdx.x & 31) == 0) {
    __threadfence();
    before = atomicAdd(reinterpret_cast<unsigned long long*>(done), 1ULL);
    __threadfence();
  }
  before = __shfl_sync(0xffffffffu, before, 0);
  __syncwarp();
  return (int64_t)before + 1 == n_ctas;
}

// Called by one warp of each of the `n_ctas` CTAs that produce results, after a CTA-wide
// barrier behind its last result or status write: the CTA that finishes last posts, so the host
// sees every CTA's words.
__device__ __forceinline__ void post_when_last(const HostPost& p, int64_t n_ctas) {
  if (!p.host) return;
  if (last_to_finish(p.done, n_ctas)) post_to_host(p);
}
#endif

// Host side of HostPost: a post for the next call on `stream` (mirroring `n_words` words from
// `dev_words`; `done_word` is a device word the call zeroes), and the wait for it.  ctx_await_post polls the pinned word, looks at the stream
// now and then (an error ends the wait; a drained stream without a post falls back to a copy),
// and leaves the words in ctx->h_words.  ctx_mark_tail records that kernels of this call may
// still be running; the next user of the context's scratch waits for them first.
HostPost ctx_begin_post(shmt_ctx* ctx, const int64_t* dev_words, int n_words, int64_t* done_word);
int ctx_await_post(shmt_ctx* ctx, const HostPost& post, cudaStream_t stream);
// A note for the next call, and the wait for it (SHMT_OK, an error, or -1: the stream has drained without it).
HostPost ctx_begin_note(shmt_ctx* ctx, int at);
int ctx_await_note(shmt_ctx* ctx, int at, cudaStream_t stream);
int ctx_mark_tail(shmt_ctx* ctx, cudaStream_t stream);
int ctx_join_tail(shmt_ctx* ctx, cudaStream_t stream);

// Device that owns a device pointer (the current device if the runtime cannot tell).
int device_of_pointer(const void* p);

// RAII device guard for entry points that are handed a context or a map.
struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  explicit DeviceGuard(int device) {
    if (cudaGetDevice(&prev) == cudaSuccess && prev != device) {
      switched = cudaSetDevice(device) == cudaSuccess;
    }
  }
  ~DeviceGuard() {
    if (switched) cudaSetDevice(prev);
  }
};

}  // namespace shmt
