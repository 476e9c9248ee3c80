// C ABI of oal_b200: argument checking, workspace carving and kernel sequencing.
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <deque>
#include <initializer_list>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "oal_intra.cuh"
#include "oal_kernels.h"
#include "oal_prologue.cuh"

namespace {

thread_local char g_error[512] = "";

int fail(int code, const char* fmt, const char* detail = "") {
  snprintf(g_error, sizeof(g_error), fmt, detail);
  return code;
}

int fail_cuda(cudaError_t e, const char* where) {
  snprintf(g_error, sizeof(g_error), "%s: %s", where, cudaGetErrorString(e));
  return OAL_ERR_CUDA;
}

// ---- launch accounting and optional per-kernel timing -----------------------------------
// Counterpart of the reference's opt-in stage profiler (oal_attention/hd_block_gemm_profiling.py):
// a launch counter that is always on, and CUDA-event pairs around every launch when enabled.
struct ProfEntry {
  const char* name;
  cudaEvent_t start, stop;
};
std::mutex g_prof_mutex;
std::vector<ProfEntry> g_prof_entries;
std::atomic<int> g_prof_enabled{0};
std::atomic<long long> g_launches{0};

struct LaunchScope {
  cudaStream_t st;
  bool timed = false;
  ProfEntry entry{};
  // `timing`: false for entry points that promise to make no allocating call (event creation is one)
  LaunchScope(const char* name, cudaStream_t stream, int launches = 1, bool timing = true) : st(stream) {
    g_launches += launches;
    if (!timing || !g_prof_enabled.load()) return;
    entry.name = name;
    if (cudaEventCreate(&entry.start) != cudaSuccess || cudaEventCreate(&entry.stop) != cudaSuccess) return;
    timed = true;
    cudaEventRecord(entry.start, st);
  }
  ~LaunchScope() {
    if (!timed) return;
    cudaEventRecord(entry.stop, st);
    std::lock_guard<std::mutex> lock(g_prof_mutex);
    g_prof_entries.push_back(entry);
  }
};

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

// ---- deferred status words ------------------------------------------------------------------
// A ring of pinned host words per device, filled by 4-byte copies on a stream of the library's own: the
// copy never sits on the caller's stream (where it would queue behind the application's own device-to-host
// copies and hold the kernels after it), and queueing one costs two event records and a copy instead of
// the tensor, stream and event objects a Python implementation creates per call.
constexpr int STATUS_RING = 1024;
struct StatusRing {
  cudaStream_t stream = nullptr;
  int32_t* host = nullptr;
  cudaEvent_t ready[STATUS_RING] = {};
  cudaEvent_t done[STATUS_RING] = {};
  long long next = 0;
};
std::mutex g_status_mutex;
StatusRing g_status[64];

// ---- delivered status words -----------------------------------------------------------------------
// A call that takes a ticket has its last kernel write the status word straight into a pinned, mapped host word: no
// copy, and a waiting host sees it a microsecond after the kernel has written it.  A ticket names a slot (word, event
// behind the call) and the slot's use.  A slot is taken again only when its call's word is in, at least
// DELIVERY_KEEP later calls have taken one, and the word has been read -- or, at the limit of slots, unread (a caller
// that never polls).  A call still in flight keeps its slot whatever the others do: a late word never lands in
// another call's ticket.
constexpr int DELIVERY_KEEP = 1024, DELIVERY_LIMIT = 4 * DELIVERY_KEEP, DELIVERY_LOOK = 64;
struct DeliverySlot {
  volatile int32_t* word = nullptr;
  cudaEvent_t done = nullptr;
  long long use = 0, taken = 0;      // uses of this slot so far; the device's count of takes at its last one
  bool recorded = false, read = false;
};
struct DeliverySlots {
  std::vector<DeliverySlot> slots;   // reserved at the first take: never moves
  std::deque<int> order;             // by take, oldest first
  int32_t* block = nullptr;          // pinned words that have no slot yet
  long long takes = 0;
};
std::mutex g_delivery_mutex;
DeliverySlots g_delivery[64];
constexpr int64_t TICKET_DELIVERED = (int64_t)1 << 62;
constexpr int TICKET_SLOT_BITS = 12;
static_assert(DELIVERY_LIMIT <= 1 << TICKET_SLOT_BITS, "slot index of a ticket");

// Calls that another thread's stream capture would not allow (event waits) in this scope.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Waits for one call's word, without any lock: on the word itself for a while (a short call is over in that time), then
// on the event behind the call -- never on the device, which may have other work queued for seconds.
cudaError_t wait_delivered(const volatile int32_t* word, cudaEvent_t done) {
  const auto t0 = std::chrono::steady_clock::now();
  for (unsigned spin = 1; !(*word & oal::STATUS_DELIVERED); ++spin)
    if ((spin & 1023) == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::milliseconds(20)) {
      if (!done) return cudaSuccess;
      RelaxedCapture scope;
      cudaError_t e;      // an event that puts the thread to sleep itself raises an interrupt in every call
      while ((e = cudaEventQuery(done)) == cudaErrorNotReady) std::this_thread::sleep_for(std::chrono::microseconds(20));
      return e;
    }
  return cudaSuccess;
}

int add_delivery_slot(DeliverySlots& d) {
  const int n = (int)d.slots.size();
  if (n == 0) d.slots.reserve(DELIVERY_LIMIT);
  if (n % DELIVERY_KEEP == 0) {
    const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&d.block), DELIVERY_KEEP * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) return fail_cuda(e, "status delivery");
  }
  DeliverySlot s;
  s.word = d.block + n % DELIVERY_KEEP;
  const cudaError_t e = cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming);
  if (e != cudaSuccess) return fail_cuda(e, "status delivery");
  d.slots.push_back(s);
  return n;
}

// A word of the current device for one call, and its ticket.
int take_delivery(int32_t** word, int64_t* ticket) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail_cuda(e, "status delivery");
  if (dev < 0 || dev >= 64) return fail(OAL_ERR_ARGUMENT, "status delivery: device index out of range");
  std::lock_guard<std::mutex> lock(g_delivery_mutex);
  DeliverySlots& d = g_delivery[dev];
  const bool at_limit = d.slots.size() == DELIVERY_LIMIT;
  int slot = -1, looked = 0;
  for (auto it = d.order.begin(); it != d.order.end() && (at_limit || looked < DELIVERY_LOOK); ++it, ++looked) {
    const DeliverySlot& s = d.slots[*it];
    if (d.takes - s.taken < DELIVERY_KEEP) break;
    if ((*s.word & oal::STATUS_DELIVERED) && (s.read || at_limit)) {
      slot = *it;
      d.order.erase(it);
      break;
    }
  }
  if (slot < 0) {
    if (at_limit) return fail(OAL_ERR_CUDA, "status delivery: too many calls in flight");
    if ((slot = add_delivery_slot(d)) < 0) return slot;
  }
  DeliverySlot& s = d.slots[slot];
  *s.word = 0;
  s.recorded = s.read = false;
  s.taken = d.takes++;
  ++s.use;
  d.order.push_back(slot);
  *word = const_cast<int32_t*>(s.word);
  *ticket = TICKET_DELIVERED | ((int64_t)dev << 48) | (int64_t)((s.use << TICKET_SLOT_BITS | slot) & (((int64_t)1 << 48) - 1));
  return OAL_OK;
}

// The slot of a ticket, or null when the slot has been taken again since; g_delivery_mutex held.
DeliverySlot* delivery_slot(int64_t ticket) {
  const int dev = (int)((ticket & ~TICKET_DELIVERED) >> 48);
  const size_t slot = (size_t)(ticket & ((1 << TICKET_SLOT_BITS) - 1));
  const long long use = (ticket & (((int64_t)1 << 48) - 1)) >> TICKET_SLOT_BITS;
  if (dev < 0 || dev >= 64 || slot >= g_delivery[dev].slots.size()) return nullptr;
  DeliverySlot& s = g_delivery[dev].slots[slot];
  return s.use == use ? &s : nullptr;
}

// After a call's last launch, or its failure: an event behind it, or a word that nothing else will write.
void finish_delivery(int64_t ticket, int rc, cudaStream_t st) {
  std::lock_guard<std::mutex> lock(g_delivery_mutex);
  DeliverySlot* s = delivery_slot(ticket);
  if (!s) return;
  if (rc) {
    *s->word = oal::STATUS_DELIVERED;
    s->read = true;
    return;
  }
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  s->recorded = cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone &&
                cudaEventRecord(s->done, st) == cudaSuccess;
}

int poll_delivery(int64_t ticket, bool block, int32_t* value) {
  constexpr const char* kExpired = "oal_status_poll: ticket expired or unknown";
  const volatile int32_t* word;
  cudaEvent_t done;
  {
    std::lock_guard<std::mutex> lock(g_delivery_mutex);
    DeliverySlot* s = delivery_slot(ticket);
    if (!s) return fail(OAL_ERR_ARGUMENT, kExpired);
    word = s->word;
    done = s->recorded ? s->done : nullptr;
  }
  if (block) {
    const cudaError_t e = wait_delivered(word, done);
    if (e != cudaSuccess) return fail_cuda(e, "oal_status_poll");
  }
  std::lock_guard<std::mutex> lock(g_delivery_mutex);
  DeliverySlot* s = delivery_slot(ticket);
  if (!s) return fail(OAL_ERR_ARGUMENT, kExpired);
  const int32_t seen = *s->word;
  if (!(seen & oal::STATUS_DELIVERED)) return block ? fail(OAL_ERR_CUDA, "oal_status_poll: the call's status word was never written") : 0;
  s->read = true;
  *value = seen & ~oal::STATUS_DELIVERED;
  return 1;
}

// ---- side streams ------------------------------------------------------------------------------
// Small kernels that nothing on the main chain waits for (the per-head factor table of the forward, the
// coefficient-gradient reductions, the reverse state scan and the whole key/value chain of the backward)
// run on two library-owned streams, forked from and joined back into the caller's stream with events, so
// every entry point still looks like work on one stream from outside (and can be captured as such).
// Streams and events are created once per device, on first use; oal_set_overlap(0) keeps everything on
// the caller's stream (the per-kernel timing of the profile report is only meaningful that way).
std::atomic<int> g_overlap{1};
struct SideStreams {
  cudaStream_t s[2] = {nullptr, nullptr};
  cudaEvent_t fork = nullptr, join[2] = {nullptr, nullptr};
  bool ok = false;
};
std::mutex g_side_mutex[64];
SideStreams g_side[64];

// `lock` is held while the call queues its forks and joins: an event that a second thread records again between a
// record and the wait that belongs to it would order the wrong streams.
SideStreams* side_streams(std::unique_lock<std::mutex>& lock) {
  if (!g_overlap.load()) return nullptr;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  lock = std::unique_lock<std::mutex>(g_side_mutex[dev]);
  SideStreams& x = g_side[dev];
  if (!x.ok) {
    bool good = cudaEventCreateWithFlags(&x.fork, cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; i < 2 && good; ++i)
      good = cudaStreamCreateWithFlags(&x.s[i], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&x.join[i], cudaEventDisableTiming) == cudaSuccess;
    if (!good) return nullptr;
    x.ok = true;
  }
  return &x;
}
// Work of one call on side stream i: starts after everything queued on `st` when it forks; mark() ends it, wait() makes
// `st` wait for that mark.  Whatever way the call is left, an error return included, the caller's stream waits: it may
// free the buffers or end a capture next.
class SideWork {
 public:
  ~SideWork() { wait(); }
  cudaStream_t fork(SideStreams* x, int i, cudaStream_t st) {
    if (!x || cudaEventRecord(x->fork, st) != cudaSuccess || cudaStreamWaitEvent(x->s[i], x->fork, 0) != cudaSuccess) return st;
    side_ = x->s[i];
    st_ = st;
    join_ = x->join[i];
    open_ = true;
    return side_;
  }
  void mark() {
    if (open_ && !marked_) marked_ = cudaEventRecord(join_, side_) == cudaSuccess;
  }
  void wait() {
    mark();
    if (open_) cudaStreamWaitEvent(st_, join_, 0);
    open_ = false;
  }

 private:
  cudaStream_t side_ = nullptr, st_ = nullptr;
  cudaEvent_t join_ = nullptr;
  bool open_ = false, marked_ = false;
};

struct Carver {
  char* base;
  size_t off = 0;
  explicit Carver(void* p) : base(static_cast<char*>(p)) {}
  template <class T>
  T* take(size_t count) {
    T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += align_up(count * sizeof(T));
    return p;
  }
};

int check_problem(const OalProblem* p) {
  if (!p) return fail(OAL_ERR_ARGUMENT, "problem is NULL");
  if (p->batch < 1 || p->q_heads < 1 || p->kv_heads < 1 || p->seq_len < 1)
    return fail(OAL_ERR_ARGUMENT, "batch, head counts and seq_len must be positive");
  if (p->q_heads % p->kv_heads) return fail(OAL_ERR_ARGUMENT, "q_heads must be divisible by kv_heads");
  if (p->head_dim != OAL_HEAD_DIM || p->value_dim != OAL_HEAD_DIM)
    return fail(OAL_ERR_ARGUMENT, "head_dim and value_dim must be 64 (the host pads smaller heads)");
  if (p->groups < 1 || p->groups > OAL_MAX_GROUPS)
    return fail(OAL_ERR_ARGUMENT, "groups must be in 1..16");
  if (p->io_dtype < 0 || p->io_dtype > 2 || p->out_dtype < 0 || p->out_dtype > 2)
    return fail(OAL_ERR_DTYPE, "io_dtype / out_dtype must be fp32, bf16 or fp16");
  if (p->precision != OAL_PRECISION_FP32_IEEE && p->precision != OAL_PRECISION_BF16_TENSORCORE)
    return fail(OAL_ERR_DTYPE, "unknown precision mode");
  if (p->precision == OAL_PRECISION_BF16_TENSORCORE) {
    if (p->io_dtype != OAL_DTYPE_BF16) return fail(OAL_ERR_DTYPE, "bf16_tensorcore requires bf16 q, k, v");
    if (p->chunk != 128) return fail(OAL_ERR_ARGUMENT, "bf16_tensorcore requires chunk == 128");
  }
  if (!(p->floor > 0.f)) return fail(OAL_ERR_ARGUMENT, "floor must be positive");
  if (p->flags & ~(OAL_FLAG_OUT_TOKEN_MAJOR | OAL_FLAG_ZERO_STATE_IN | OAL_FLAG_NO_BACKWARD)) return fail(OAL_ERR_ARGUMENT, "unknown bits in flags");
  if ((p->flags & OAL_FLAG_OUT_TOKEN_MAJOR) && (p->precision != OAL_PRECISION_BF16_TENSORCORE || p->groups > 8))
    // (the limit of 8 groups is the flag's contract; the kernels have none)
    return fail(OAL_ERR_ARGUMENT, "token-major out needs bf16_tensorcore and at most 8 groups per head");
  return OAL_OK;
}

// The tensor-core kernels and the row moves read and write these tensors in 16-byte pieces.  (The exact fp32 kernels
// look at the alignment themselves and fall back to single elements; they ask it of the workspace only.)
bool misaligned(std::initializer_list<const void*> tensors) {
  uintptr_t bits = 0;
  for (const void* t : tensors) bits |= reinterpret_cast<uintptr_t>(t);
  return bits & 15;
}
constexpr const char* kMisaligned = "%s: tensors must start on a 16-byte boundary";

// Where a call's coefficients come from: the packed factor (expanded on the device into A, B, C), or A, B, C.
struct CoefSource {
  const float* factor;      // null: A, B, C are inputs
  int factor_rows;
  float eps;
  float *A, *B, *C;
};

CoefSource explicit_coefs(const float* a, const float* b, const float* c) {
  return CoefSource{nullptr, 0, 0.f, const_cast<float*>(a), const_cast<float*>(b), const_cast<float*>(c)};
}
CoefSource packed_coefs(const OalProblem* p, const float* factor, int factor_rows, float eps, float* coefs) {
  float* b = coefs + p->q_heads;
  return CoefSource{factor, factor_rows, eps, coefs, b, b + (size_t)p->q_heads * p->groups};
}

// Gradient of the coefficients: dA, dB, dC, and the packed factor's when it was the source.
struct CoefSink {
  float *dA, *dB, *dC, *dfactor;
};

oal::PrologueArgs prologue_args(const OalProblem* p, const CoefSource& src, const int32_t* dim_perm, const int32_t* group_start,
                                float* coef_table, void* factors, int32_t* status, int32_t* counter) {
  return oal::PrologueArgs{src.factor, src.factor_rows, p->groups, src.eps, p->scale, dim_perm, group_start, src.A, src.B, src.C,
                           coef_table, static_cast<oal::HeadFactor*>(factors), status, counter};
}

struct BackwardSpace {
  float* g;
  float* coef_pairs;
  float* dcoefs;
  float *dk_part, *dv_part;
  size_t bytes;
};

int coef_slots_pairs(const OalProblem* p) {
  return oal::pairs_tiles(p->seq_len) * oal::pairs_split(p->batch, p->q_heads, p->seq_len);
}

size_t coef_floats(const OalProblem* p) { return (size_t)p->q_heads * (1 + p->groups + p->groups * p->groups); }

BackwardSpace carve_backward(const OalProblem* p, void* ws) {
  Carver c(ws);
  BackwardSpace s;
  const size_t rows = (size_t)p->batch * p->q_heads * p->seq_len;
  s.g = c.take<float>(rows * oal::EP);
  s.coef_pairs = c.take<float>((size_t)p->batch * p->q_heads * coef_slots_pairs(p) * oal::NCOEF);
  s.dcoefs = c.take<float>(coef_floats(p));
  const size_t shares = p->q_heads > p->kv_heads ? rows * oal::HD : 0;
  s.dk_part = c.take<float>(shares);
  s.dv_part = c.take<float>(shares);
  s.bytes = c.off;
  return s;
}

constexpr int kChunk = 128;

int chunk_count(const OalProblem* p) { return (p->seq_len + kChunk - 1) / kChunk; }

// Chunks that meet a state.  Without a state from earlier tokens the first chunk of a sequence reads none and
// nothing needs the increment of the last one, and the other way round in the backward: a share of 1 / chunks of
// the state work, all of it for a sequence of one chunk.
struct ChunkRange {
  bool trim;
  int n;         // chunks that read a state: the last n (forward), the first n (key side of the backward)
  int first;     // first chunk that reads a carry
};
ChunkRange chunk_range(const OalProblem* p, const void* state_in, const void* dstate_in) {
  const bool trim = (p->flags & OAL_FLAG_ZERO_STATE_IN) && !state_in && !dstate_in && !(p->grad_mask & OAL_GRAD_REUSE_STATE_STAGE);
  const int nb = chunk_count(p);
  return ChunkRange{trim, trim ? nb - 1 : nb, trim ? 1 : 0};
}

struct ForwardSpaceTC {
  float* ds;
  size_t bytes;
};

int make_head_factors(const OalProblem* p, const int32_t* dim_perm, const int32_t* group_start, const float* coef_a,
                      const float* coef_b, const float* coef_c, void* factors, cudaStream_t st, bool timing = true) {
  LaunchScope scope("head_factors", st, 1, timing);
  cudaError_t e = oal::build_head_factors(dim_perm, group_start, coef_a, coef_b, coef_c, p->q_heads, p->groups,
                                          p->scale, factors, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "head factor kernel");
}

ForwardSpaceTC carve_forward_tc(const OalProblem* p, void* ws) {
  Carver c(ws);
  ForwardSpaceTC s;
  const size_t units = (size_t)p->batch * p->kv_heads;
  s.ds = c.take<float>(units * chunk_count(p) * oal::state_rows() * oal::EP);
  s.bytes = c.off;
  return s;
}

// The buffer the forward hands to the backward: the bf16 carry images of every chunk (the MMA operand),
// the images of their rounding remainders (read only by the coefficient-gradient dot products), then the
// per-head factor table of the intra-chunk kernels and the per-feature coefficient table of the state kernels
// (the backward of the same call sees the same coefficients), then the images of the rows of k and [v | 1].
size_t saved_images_bytes_tc(const OalProblem* p) {
  return align_up((size_t)p->batch * p->kv_heads * chunk_count(p) * oal::state_image_bytes_per_chunk());
}
size_t saved_factors_bytes_tc(const OalProblem* p) { return align_up(oal::head_factor_bytes(p->q_heads)); }
size_t saved_rows_offset_tc(const OalProblem* p) {
  return 2 * saved_images_bytes_tc(p) + saved_factors_bytes_tc(p) + align_up((size_t)p->q_heads * oal::state_rows() * sizeof(float));
}
size_t k_image_bytes_tc(const OalProblem* p) { return align_up((size_t)p->batch * p->kv_heads * chunk_count(p) * oal::ROW_IMAGE_BYTES); }
size_t saved_state_bytes_tc(const OalProblem* p) {
  return saved_rows_offset_tc(p) + k_image_bytes_tc(p) + align_up((size_t)p->batch * p->kv_heads * chunk_count(p) * oal::state_slab_image_bytes());
}
char* saved_at(const void* saved_state, size_t offset) {
  return const_cast<char*>(static_cast<const char*>(saved_state)) + offset;
}
void* saved_remainders(const OalProblem* p, const void* saved_state) { return saved_at(saved_state, saved_images_bytes_tc(p)); }
void* saved_factors(const OalProblem* p, const void* saved_state) { return saved_at(saved_state, 2 * saved_images_bytes_tc(p)); }
float* saved_coef_table(const OalProblem* p, const void* saved_state) {
  return reinterpret_cast<float*>(saved_at(saved_state, 2 * saved_images_bytes_tc(p) + saved_factors_bytes_tc(p)));
}

oal::RowImages row_images(const OalProblem* p, const void* saved_state, const void* q, const void* k, const void* v, void* q_image) {
  char* rows = saved_at(saved_state, saved_rows_offset_tc(p));
  return oal::RowImages{q, k, v, q_image, rows, rows + k_image_bytes_tc(p)};
}

struct BackwardSpaceTC {
  float* coef_blocks;            // coefficient partial sums of the query row blocks
  void* gimg;
  void* q_image;                 // rows of q as operand images
  float* dcarry;
  void* dt_img;
  float* dcoef_partial;
  float* dcoef;
  float* slots;
  float *dq_cross, *dk_cross, *dv_cross;
  float *dk_part, *dv_part;      // shares of dk / dv of groups of query heads
  float* dcoefs;                 // dA, dB, dC of a call whose caller asks for the factor's gradient
  size_t bytes;
};

BackwardSpaceTC carve_backward_tc(const OalProblem* p, void* ws) {
  Carver c(ws);
  BackwardSpaceTC s;
  const size_t units = (size_t)p->batch * p->kv_heads, nb = chunk_count(p);
  const size_t qrows = (size_t)p->batch * p->q_heads * p->seq_len;
  const size_t krows = (size_t)p->batch * p->kv_heads * p->seq_len;
  const size_t slab_image = oal::state_slab_image_bytes();
  s.coef_blocks = c.take<float>((size_t)p->batch * p->q_heads * oal::intra_row_blocks(p->seq_len) * (1 + p->groups + p->groups * (p->groups + 1) / 2));
  s.gimg = c.take<char>(2 * (size_t)p->batch * p->q_heads * nb * slab_image);   // hi image, then lo image
  s.q_image = c.take<char>((size_t)p->batch * p->q_heads * nb * oal::ROW_IMAGE_BYTES);
  s.dcarry = c.take<float>(units * nb * oal::state_rows() * oal::EP);
  s.dt_img = c.take<char>(units * nb * oal::state_image_bytes_per_chunk());
  s.dcoef_partial = c.take<float>(2 * (size_t)p->batch * nb * p->q_heads * oal::state_rows());   // two column halves
  s.dcoef = c.take<float>((size_t)p->q_heads * oal::state_rows());
  s.slots = c.take<float>((size_t)p->q_heads * oal::NCOEF);
  s.dq_cross = c.take<float>(qrows * oal::HD);
  s.dk_cross = c.take<float>(krows * oal::HD);
  s.dv_cross = c.take<float>(krows * oal::VD);
  s.dk_part = c.take<float>(qrows * oal::HD);
  s.dv_part = c.take<float>(qrows * oal::VD);
  s.dcoefs = c.take<float>(coef_floats(p));
  s.bytes = c.off;
  return s;
}

// Stage A of the tensor-core backward: everything that does not depend on later tokens' state
// gradient (normalisation VJP, per-chunk dCarry and coefficient partial sums).
int backward_vjp(const OalProblem* p, const float* num, const float* den, const void* grad_out, const float* grad_num,
                 const float* grad_den, const BackwardSpaceTC& s, const oal::RowImages& rows, int32_t* clear_status, cudaStream_t st) {
  LaunchScope scope("norm_vjp", st);
  const cudaError_t e = oal::norm_vjp_image(grad_out, p->out_dtype, grad_num, grad_den, num, den, p->floor, s.gimg,
                                            p->batch * p->q_heads, p->seq_len, chunk_count(p),
                                            (p->flags & OAL_FLAG_OUT_TOKEN_MAJOR) ? p->q_heads : 0, rows, clear_status, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "normalisation VJP kernel");
}
int backward_dstate(const OalProblem* p, const void* saved_state, const ChunkRange& cr, const BackwardSpaceTC& s,
                    int32_t* status, cudaStream_t st) {
  const bool want_c = p->grad_mask & OAL_GRAD_COEF;
  if (!(p->grad_mask & (OAL_GRAD_K | OAL_GRAD_V | OAL_GRAD_COEF)) || cr.n == 0) return OAL_OK;
  LaunchScope scope("dstate_heads", st);
  const cudaError_t e = oal::dstate_heads(s.q_image, s.gimg, want_c ? saved_state : nullptr,
                                          want_c ? saved_remainders(p, saved_state) : nullptr, saved_coef_table(p, saved_state),
                                          s.dcarry, want_c ? s.dcoef_partial : nullptr, p->batch, p->q_heads, p->kv_heads,
                                          chunk_count(p), cr.first, cr.n, p->scale, status, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "state gradient kernel");
}

oal::PairArgs base_args(const OalProblem* p, const void* q, const void* k, const void* v,
                        const int32_t* perm, const int32_t* gstart, const CoefSource& src, int32_t* status) {
  oal::PairArgs a;
  memset(&a, 0, sizeof(a));
  a.B = p->batch; a.Hq = p->q_heads; a.Hkv = p->kv_heads; a.N = p->seq_len; a.G = p->groups;
  a.io_dt = p->io_dtype; a.out_dt = p->out_dtype;
  a.scale = p->scale; a.floor = p->floor;
  a.q = q; a.k = k; a.v = v;
  a.dim_perm = perm; a.group_start = gstart;
  a.A = src.A; a.Bc = src.B; a.Cc = src.C;
  a.status = status;
  return a;
}

// ---- forward ------------------------------------------------------------------------------------
int forward_core(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                 const int32_t* group_start, const CoefSource& src, void* out, float* num, float* den, void* saved_state,
                 const float* state_in, float* ds, int32_t* status, oal::StatusSink sink, bool timing,
                 cudaStream_t st) {
  cudaError_t e;
  const bool tc = p->precision == OAL_PRECISION_BF16_TENSORCORE;
  const int units = p->batch * p->kv_heads, nb = chunk_count(p);
  const ChunkRange cr = chunk_range(p, state_in, nullptr);
  const bool reuse = p->grad_mask & OAL_GRAD_REUSE_STATE_STAGE;      // increments left by oal_forward_local_state
  const bool update = tc && !reuse && cr.n > 0;
  void* factors = tc ? saved_factors(p, saved_state) : nullptr;
  float* coef_table = tc ? saved_coef_table(p, saved_state) : nullptr;
  std::unique_lock<std::mutex> side_lock;
  SideStreams* side = nullptr;
  SideWork beside;
  cudaStream_t s0 = st;
  oal::PrologueArgs pro{};
  const oal::RowImages rows = tc ? row_images(p, saved_state, q, k, v, nullptr) : oal::RowImages{};
  if (src.factor) {
    pro = prologue_args(p, src, dim_perm, group_start, coef_table, factors, status, sink.host ? sink.counter : nullptr);
    if (!tc) {
      LaunchScope scope("head_prologue", st, 1, timing);
      if ((e = oal::launch_head_prologue(pro, p->q_heads, st)) != cudaSuccess) return fail_cuda(e, "prologue kernel");
    } else if (cr.n > 0 && timing && (side = side_streams(side_lock))) {
      // The rotations (11 us at 8 groups, 45 at 16) are needed by the call's last kernel only, the coefficients by the
      // next but one: with both in one launch the state kernels waited for the rotations.  Beside the state
      // kernels they cost the host a launch and two events.  14 / 2 heads, B = 1, both forms in us: forward + backward
      // N = 256 169 -> 160, N = 1024 198 -> 190, replayed 203 -> 192, 16 groups N = 4096 663 -> 647.
      s0 = beside.fork(side, 0, st);
      oal::PrologueArgs own = pro;
      own.A = own.B = own.C = own.coef_table = nullptr;
      own.status = own.counter = nullptr;
      pro.factors = nullptr;
      LaunchScope scope("head_prologue", s0, 1, timing);
      if ((e = oal::launch_head_prologue(own, p->q_heads, s0)) != cudaSuccess) return fail_cuda(e, "prologue kernel");
      beside.mark();
    }
  } else if (tc) {
    // explicit coefficients: the factor table (rotations of a possibly indefinite matrix, 50 us) is needed by the
    // last kernel only and is computed beside the state kernels
    if (timing) side = side_streams(side_lock);
    s0 = beside.fork(side, 0, st);
    if (int rc = make_head_factors(p, dim_perm, group_start, src.A, src.B, src.C, factors, s0, timing)) return rc;
    beside.mark();
    LaunchScope scope("coef_table", st, 1, timing);
    e = oal::build_coef_table(dim_perm, group_start, src.A, src.B, src.C, p->q_heads, p->groups, p->scale, coef_table, st);
    if (e != cudaSuccess) return fail_cuda(e, "coefficient table kernel");
  }
  const bool walk = update && oal::state_walk_pays(units, nb);
  const bool backward = !(p->flags & OAL_FLAG_NO_BACKWARD);
  if (tc && (src.factor || walk || backward)) {
    LaunchScope scope("rows_prologue", st, 1, timing);
    e = oal::rows_prologue(rows, walk || backward ? units : 0, p->seq_len, nb, src.factor ? &pro : nullptr, p->q_heads, st);
    if (e != cudaSuccess) return fail_cuda(e, "row image kernel");
  }
  void* remainders = tc && backward ? saved_remainders(p, saved_state) : nullptr;
  if (walk) {
    LaunchScope scope("state_walk", st, 1, timing);
    e = oal::state_walk(rows, saved_state, remainders, state_in, units, nb, cr.trim, status, st);
    if (e != cudaSuccess) return fail_cuda(e, "state walk kernel");
  } else if (update) {
    LaunchScope scope("state_update", st, 1, timing);
    e = oal::state_update(k, v, ds, units, p->seq_len, nb, cr.n, status, st);
    if (e != cudaSuccess) return fail_cuda(e, "state update kernel");
  }
  if (tc && cr.n > 0) {
    if (!walk) {
      LaunchScope scope("state_scan", st, 1, timing);
      e = oal::state_scan(ds, saved_state, remainders, state_in, nullptr, units, nb, 0, cr.trim, st);
      if (e != cudaSuccess) return fail_cuda(e, "state scan kernel");
    }
    { LaunchScope scope("cross_read_q", st, 1, timing);
      e = oal::cross_read(true, q, saved_state, coef_table, num, den, p->batch, p->q_heads, p->q_heads / p->kv_heads,
                          p->seq_len, nb, cr.first, cr.n, status, st); }
    if (e != cudaSuccess) return fail_cuda(e, "cross read kernel");
  }
  if (tc) {
    beside.wait();
    LaunchScope scope("intra_forward", st, 1, timing);
    e = oal::intra_forward(q, k, v, factors, out, num, den, status, p->batch, p->q_heads, p->kv_heads, p->seq_len, nb, p->groups,
                           p->out_dtype, p->floor, (p->flags & OAL_FLAG_OUT_TOKEN_MAJOR) != 0, cr.first, sink, st);
    return e == cudaSuccess ? OAL_OK : fail_cuda(e, "intra-chunk forward kernel");
  }
  oal::PairArgs a = base_args(p, q, k, v, dim_perm, group_start, src, status);
  a.out = out; a.num = num; a.den = den;
  a.sink = sink;
  LaunchScope scope("pairs_forward", st, 1, timing);
  e = oal::pairs_forward(a, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "forward pair kernel");
}

// ---- backward -----------------------------------------------------------------------------------
// sums of the coefficient partials -> dA, dB, dC, and on to the packed factor
int finish_coefs(const OalProblem* p, const CoefSource& src, const CoefSink& sink, const float* partial, const float* slots,
                 bool chunked, cudaStream_t st) {
  cudaError_t e;
  const bool fused = chunked && sink.dfactor && src.factor_rows == p->q_heads;
  { LaunchScope scope("reduce_coefs", st);
    e = chunked ? oal::intra_coef_finish(partial, oal::intra_row_blocks(p->seq_len), slots, p->batch, p->q_heads, p->groups, sink.dA,
                                         sink.dB, sink.dC, fused ? src.factor : nullptr, fused ? sink.dfactor : nullptr, st)
                : oal::reduce_coefs(partial, coef_slots_pairs(p), slots, p->batch, p->q_heads, p->groups,
                                    sink.dA, sink.dB, sink.dC, st); }
  if (e != cudaSuccess) return fail_cuda(e, "coefficient reduction kernel");
  if (sink.dfactor && !fused) {
    LaunchScope scope("expand_factor_grad", st);
    e = oal::expand_factor_grad(src.factor, src.factor_rows, p->q_heads, p->groups, sink.dA, sink.dB, sink.dC, sink.dfactor, st);
    if (e != cudaSuccess) return fail_cuda(e, "factor gradient kernel");
  }
  return OAL_OK;
}

struct BackwardArgs {
  const void *q, *k, *v;
  const int32_t *dim_perm, *group_start;
  const float *num, *den;
  const void *saved_state, *grad_out;
  const float *grad_num, *grad_den;
  void *dq, *dk, *dv;
  const float* dstate_in;
  void* workspace;
  size_t workspace_bytes;
  int32_t* status;
  bool clear_status;          // the first kernel zeroes the word
};

int backward_core_fp32(const OalProblem* p, const BackwardArgs& x, const CoefSource& src, CoefSink sink, cudaStream_t st) {
  if (x.dstate_in) return fail(OAL_ERR_ARGUMENT, "fp32_ieee mode keeps no chunk state: dstate_in must be NULL");
  BackwardSpace s = carve_backward(p, x.workspace);
  if (!x.workspace || x.workspace_bytes < s.bytes) return fail(OAL_ERR_WORKSPACE, "oal_backward: workspace too small");
  if (misaligned({x.workspace})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_backward");
  const int mask = p->grad_mask;
  if (sink.dfactor) {
    sink.dA = s.dcoefs; sink.dB = sink.dA + p->q_heads; sink.dC = sink.dB + (size_t)p->q_heads * p->groups;
  }
  const size_t rows = (size_t)p->batch * p->q_heads * p->seq_len;
  cudaError_t e;
  { LaunchScope scope("norm_vjp", st);
    e = oal::norm_vjp(x.grad_out, p->out_dtype, x.grad_num, x.grad_den, x.num, x.den, p->floor, s.g, rows,
                      x.clear_status ? x.status : nullptr, st); }
  if (e != cudaSuccess) return fail_cuda(e, "normalisation VJP kernel");
  oal::PairArgs a = base_args(p, x.q, x.k, x.v, x.dim_perm, x.group_start, src, x.status);
  a.g = s.g;
  const bool want_kv = mask & (OAL_GRAD_K | OAL_GRAD_V);
  // The two sides share no buffer: the key/value side fills the SMs that the last blocks of the query side leave idle
  // (all but a few SMs in a short call).
  std::unique_lock<std::mutex> side_lock;
  SideStreams* side = side_streams(side_lock);
  SideWork kv;
  cudaStream_t skv = want_kv ? kv.fork(side, 0, st) : st;
  if (mask & (OAL_GRAD_Q | OAL_GRAD_COEF)) {
    a.dq = (mask & OAL_GRAD_Q) ? x.dq : nullptr;
    a.coef_partial = (mask & OAL_GRAD_COEF) ? s.coef_pairs : nullptr;
    { LaunchScope scope("pairs_backward_q", st); e = oal::pairs_backward_q(a, st); }
    if (e != cudaSuccess) return fail_cuda(e, "backward query-side pair kernel");
  }
  if (want_kv) {
    a.dq = nullptr; a.coef_partial = nullptr;
    a.dk_part = s.dk_part; a.dv_part = s.dv_part;
    a.dk = (mask & OAL_GRAD_K) ? x.dk : nullptr;
    a.dv = (mask & OAL_GRAD_V) ? x.dv : nullptr;
    { LaunchScope scope("pairs_backward_kv", skv, p->q_heads > p->kv_heads ? 2 : 1); e = oal::pairs_backward_kv(a, skv); }
    if (e != cudaSuccess) return fail_cuda(e, "backward key/value-side pair kernels");
    kv.mark();
  }
  if (mask & OAL_GRAD_COEF)
    if (int rc = finish_coefs(p, src, sink, s.coef_pairs, nullptr, false, st)) return rc;
  kv.wait();
  return OAL_OK;
}

int backward_core(const OalProblem* p, const BackwardArgs& x, const CoefSource& src, CoefSink sink, cudaStream_t st) {
  if (p->flags & OAL_FLAG_NO_BACKWARD) return fail(OAL_ERR_ARGUMENT, "oal_backward: the problem says that no backward follows");
  if (p->precision == OAL_PRECISION_FP32_IEEE) return backward_core_fp32(p, x, src, sink, st);
  if (!x.saved_state) return fail(OAL_ERR_ARGUMENT, "oal_backward: saved_state is NULL");
  if (misaligned({x.q, x.k, x.v, x.num, x.saved_state, x.grad_out, x.grad_num, x.dq, x.dk, x.dv, x.dstate_in, x.workspace}))
    return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_backward");
  BackwardSpaceTC s = carve_backward_tc(p, x.workspace);
  if (!x.workspace || x.workspace_bytes < s.bytes) return fail(OAL_ERR_WORKSPACE, "oal_backward: workspace too small");
  if (sink.dfactor) {
    sink.dA = s.dcoefs; sink.dB = sink.dA + p->q_heads; sink.dC = sink.dB + (size_t)p->q_heads * p->groups;
  }
  const int mask = p->grad_mask;
  const int nb = chunk_count(p), units = p->batch * p->kv_heads, rep = p->q_heads / p->kv_heads;
  const bool want_q = mask & OAL_GRAD_Q, want_k = mask & OAL_GRAD_K, want_v = mask & OAL_GRAD_V, want_kv = want_k || want_v;
  const bool want_c = mask & OAL_GRAD_COEF;
  const bool reuse = mask & OAL_GRAD_REUSE_STATE_STAGE;
  const ChunkRange cr = chunk_range(p, nullptr, x.dstate_in);
  const void* factors = saved_factors(p, x.saved_state);      // written by the forward of this call
  const float* coef_table = saved_coef_table(p, x.saved_state);
  const oal::RowImages rows = row_images(p, x.saved_state, x.q, x.k, x.v, s.q_image);
  cudaError_t e;
  if (!reuse) {
    if (int rc = backward_vjp(p, x.num, x.den, x.grad_out, x.grad_num, x.grad_den, s, rows, x.clear_status ? x.status : nullptr, st)) return rc;
    if (int rc = backward_dstate(p, x.saved_state, cr, s, x.status, st)) return rc;
  }
  // Three chains leave the state stage: the query side (on the caller's stream), the key/value side and
  // the reduction of the cross-chunk coefficient gradient.  They share no buffer, so the last two run on
  // the library's side streams and are joined before this function returns.
  std::unique_lock<std::mutex> side_lock;
  SideStreams* side = side_streams(side_lock);
  const bool cross = cr.n > 0;
  SideWork kv, cross_coefs;
  cudaStream_t skv = want_kv ? kv.fork(side, 0, st) : st;
  cudaStream_t sc = want_c && cross ? cross_coefs.fork(side, 1, st) : st;
  if (want_c && cross) {
    { LaunchScope scope("dcoef_reduce", sc, 2);
      e = oal::dcoef_reduce(s.dcoef_partial, 2 * p->batch * cr.n, p->q_heads, p->groups, x.dim_perm, x.group_start, s.dcoef, s.slots, sc); }
    if (e != cudaSuccess) return fail_cuda(e, "coefficient gradient reduction kernels");
    cross_coefs.mark();
  }
  if (want_kv && cross) {
    { LaunchScope scope("state_scan_reverse", skv);
      e = oal::state_scan(s.dcarry, s.dt_img, nullptr, x.dstate_in, nullptr, units, nb, 1, cr.trim, skv); }
    if (e != cudaSuccess) return fail_cuda(e, "reverse state scan kernel");
    if (want_k) {
      { LaunchScope scope("feature_grad_k", skv);
        e = oal::feature_grad(false, rows.k_image, rows.u_image, s.dt_img, nullptr, s.dk_cross, p->batch, p->kv_heads, 1,
                              p->seq_len, nb, 0, cr.n, x.status, skv); }
      if (e != cudaSuccess) return fail_cuda(e, "key feature gradient kernel");
    }
    if (want_v) {
      { LaunchScope scope("cross_read_k", skv);
        e = oal::cross_read(false, x.k, s.dt_img, nullptr, s.dv_cross, nullptr, p->batch, p->kv_heads, 1, p->seq_len,
                            nb, 0, cr.n, x.status, skv); }
      if (e != cudaSuccess) return fail_cuda(e, "key cross read kernel");
    }
  }
  if (want_q && cross) {
    { LaunchScope scope("feature_grad_q", st);
      e = oal::feature_grad(true, s.q_image, s.gimg, x.saved_state, coef_table, s.dq_cross, p->batch, p->q_heads,
                            rep, p->seq_len, nb, cr.first, cr.n, x.status, st); }
    if (e != cudaSuccess) return fail_cuda(e, "query feature gradient kernel");
  }
  if (want_q || want_c) {
    { LaunchScope scope("intra_backward_q", st);
      e = oal::intra_backward_q(rows, s.gimg, factors, want_q ? x.dq : nullptr, want_q ? s.dq_cross : nullptr,
                                want_c ? s.coef_blocks : nullptr, x.status, p->batch, p->q_heads, p->kv_heads,
                                p->seq_len, nb, p->groups, p->scale, cr.first, st); }
    if (e != cudaSuccess) return fail_cuda(e, "intra-chunk backward query-side kernel");
  }
  if (want_kv) {
    // the two intra-chunk kernels each fill the machine: the key/value one is queued after the query one
    { LaunchScope scope("intra_backward_kv", skv, oal::intra_kv_parts(p->batch, p->q_heads, p->kv_heads, nb) > 1 ? 2 : 1);
      e = oal::intra_backward_kv(rows, s.gimg, factors, want_k ? x.dk : nullptr, want_v ? x.dv : nullptr, s.dk_cross,
                                 s.dv_cross, cr.n * kChunk, s.dk_part, s.dv_part, x.status, p->batch, p->q_heads, p->kv_heads,
                                 p->seq_len, nb, p->groups, skv); }
    if (e != cudaSuccess) return fail_cuda(e, "intra-chunk backward key/value-side kernels");
    kv.mark();
  }
  if (want_c) {
    cross_coefs.wait();
    if (int rc = finish_coefs(p, src, sink, s.coef_blocks, cross ? s.slots : nullptr, true, st)) return rc;
  }
  kv.wait();
  return OAL_OK;
}

}  // namespace

extern "C" {

int oal_rope_pack(const void* q_flat, const void* k_flat, const void* v_flat, const float* cosv, const float* sinv,
                  void* q, void* k, void* v, int batch, int seq_len, int q_heads, int kv_heads, void* stream) {
  if (batch < 0 || seq_len < 0 || q_heads < 1 || kv_heads < 1) return fail(OAL_ERR_ARGUMENT, "oal_rope_pack: bad geometry");
  if ((q_flat || k_flat) && (!cosv || !sinv)) return fail(OAL_ERR_ARGUMENT, "oal_rope_pack: cos / sin are required");
  if (misaligned({q_flat, k_flat, v_flat, cosv, sinv, q, k, v})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_rope_pack");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  LaunchScope scope("rope_pack", st, (q_flat ? 1 : 0) + (k_flat ? 1 : 0) + (v_flat ? 1 : 0));
  if (q_flat && (e = oal::rope_to_heads(q_flat, q, cosv, sinv, batch, seq_len, q_heads, true, st)) != cudaSuccess)
    return fail_cuda(e, "rotary pack kernel (q)");
  if (k_flat && (e = oal::rope_to_heads(k_flat, k, cosv, sinv, batch, seq_len, kv_heads, true, st)) != cudaSuccess)
    return fail_cuda(e, "rotary pack kernel (k)");
  if (v_flat && (e = oal::rope_to_heads(v_flat, v, nullptr, nullptr, batch, seq_len, kv_heads, false, st)) != cudaSuccess)
    return fail_cuda(e, "pack kernel (v)");
  return OAL_OK;
}

int oal_rope_unpack_grad(const void* dq, const void* dk, const void* dv, const float* cosv, const float* sinv,
                         void* dq_flat, void* dk_flat, void* dv_flat, int batch, int seq_len, int q_heads,
                         int kv_heads, void* stream) {
  if (batch < 0 || seq_len < 0 || q_heads < 1 || kv_heads < 1)
    return fail(OAL_ERR_ARGUMENT, "oal_rope_unpack_grad: bad geometry");
  if ((dq || dk) && (!cosv || !sinv)) return fail(OAL_ERR_ARGUMENT, "oal_rope_unpack_grad: cos / sin are required");
  if (misaligned({dq, dk, dv, cosv, sinv, dq_flat, dk_flat, dv_flat})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_rope_unpack_grad");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  LaunchScope scope("rope_unpack_grad", st, (dq ? 1 : 0) + (dk ? 1 : 0) + (dv ? 1 : 0));
  if (dq && (e = oal::rope_to_flat(dq, dq_flat, cosv, sinv, batch, seq_len, q_heads, true, st)) != cudaSuccess)
    return fail_cuda(e, "rotary unpack kernel (dq)");
  if (dk && (e = oal::rope_to_flat(dk, dk_flat, cosv, sinv, batch, seq_len, kv_heads, true, st)) != cudaSuccess)
    return fail_cuda(e, "rotary unpack kernel (dk)");
  if (dv && (e = oal::rope_to_flat(dv, dv_flat, nullptr, nullptr, batch, seq_len, kv_heads, false, st)) != cudaSuccess)
    return fail_cuda(e, "unpack kernel (dv)");
  return OAL_OK;
}

const char* oal_last_error_string(void) { return g_error; }

const char* oal_version_string(void) { return "oal_b200 0.1 sm_100a"; }

int64_t oal_launch_count(void) { return g_launches.load(); }

void oal_profile_enable(int enable) {
  std::lock_guard<std::mutex> lock(g_prof_mutex);
  for (auto& e : g_prof_entries) {
    cudaEventDestroy(e.start);
    cudaEventDestroy(e.stop);
  }
  g_prof_entries.clear();
  g_prof_enabled.store(enable ? 1 : 0);
}

int oal_profile_report(char* buffer, size_t capacity) {
  std::lock_guard<std::mutex> lock(g_prof_mutex);
  std::map<std::string, std::pair<int, double>> agg;
  for (auto& e : g_prof_entries) {
    if (cudaEventSynchronize(e.stop) != cudaSuccess) return fail(OAL_ERR_CUDA, "oal_profile_report: event synchronise failed");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e.start, e.stop);
    auto& slot = agg[e.name];
    slot.first += 1;
    slot.second += ms;
    cudaEventDestroy(e.start);
    cudaEventDestroy(e.stop);
  }
  g_prof_entries.clear();
  std::string out = "{";
  bool first = true;
  for (auto& kv : agg) {
    char item[160];
    snprintf(item, sizeof(item), "%s\"%s\": [%d, %.6f]", first ? "" : ", ", kv.first.c_str(), kv.second.first,
             kv.second.second);
    out += item;
    first = false;
  }
  out += "}";
  if (!buffer || out.size() + 1 > capacity) return fail(OAL_ERR_ARGUMENT, "oal_profile_report: buffer too small");
  memcpy(buffer, out.c_str(), out.size() + 1);
  return OAL_OK;
}

int64_t oal_workspace_bytes(const OalProblem* p, int phase) {
  int rc = check_problem(p);
  if (rc) return rc;
  if (phase < 0 || phase > 2) return fail(OAL_ERR_ARGUMENT, "phase must be 0 (forward), 1 (backward) or 2 (saved state)");
  if (p->precision == OAL_PRECISION_FP32_IEEE) {
    if (phase == 1) return (int64_t)carve_backward(p, nullptr).bytes;
    return 0;
  }
  if (phase == 0) return (int64_t)carve_forward_tc(p, nullptr).bytes;
  if (phase == 2) return (int64_t)saved_state_bytes_tc(p);
  return (int64_t)carve_backward_tc(p, nullptr).bytes;
}

static int forward_entry(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                         const int32_t* group_start, const CoefSource& src, void* out, float* num, float* den, void* saved_state,
                         const float* state_in, void* workspace, size_t workspace_bytes, int32_t* status, oal::StatusSink sink,
                         void* stream) {
  if (!q || !k || !v || !dim_perm || !group_start || !src.A || !src.B || !src.C || !out || !num || !den || !status)
    return fail(OAL_ERR_ARGUMENT, "oal_forward: NULL tensor pointer");
  float* ds = nullptr;
  if (p->precision == OAL_PRECISION_FP32_IEEE) {
    if (state_in) return fail(OAL_ERR_ARGUMENT, "fp32_ieee mode keeps no chunk state: state_in must be NULL");
  } else {
    if (misaligned({q, k, v, out, num, saved_state, state_in, workspace})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_forward");
    ForwardSpaceTC s = carve_forward_tc(p, workspace);
    if (!workspace || workspace_bytes < s.bytes) return fail(OAL_ERR_WORKSPACE, "oal_forward: workspace too small");
    if (!saved_state) return fail(OAL_ERR_ARGUMENT, "oal_forward: saved_state is NULL");
    ds = s.ds;
  }
  return forward_core(p, q, k, v, dim_perm, group_start, src, out, num, den, saved_state, state_in, ds, status, sink, true,
                      static_cast<cudaStream_t>(stream));
}

int oal_forward(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                const int32_t* group_start, const float* coef_a, const float* coef_b, const float* coef_c,
                void* out, float* num, float* den, void* saved_state, const float* state_in,
                void* workspace, size_t workspace_bytes, int32_t* status, void* stream) {
  if (int rc = check_problem(p)) return rc;
  return forward_entry(p, q, k, v, dim_perm, group_start, explicit_coefs(coef_a, coef_b, coef_c), out, num, den, saved_state,
                       state_in, workspace, workspace_bytes, status, oal::StatusSink{nullptr, nullptr}, stream);
}

int oal_forward_packed(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                       const int32_t* group_start, const float* factor, int factor_rows, float kernel_eps, float* coefs, void* out,
                       float* num, float* den, void* saved_state, void* workspace, size_t workspace_bytes, int32_t* status,
                       int64_t* ticket, void* stream) {
  if (int rc = check_problem(p)) return rc;
  if (!factor || !coefs) return fail(OAL_ERR_ARGUMENT, "oal_forward_packed: NULL pointer");
  if (factor_rows != 1 && factor_rows != p->q_heads) return fail(OAL_ERR_ARGUMENT, "oal_forward_packed: factor_rows must be 1 or q_heads");
  oal::StatusSink sink{nullptr, nullptr};
  if (ticket) {
    int32_t* word = nullptr;
    if (int rc = take_delivery(&word, ticket)) return rc;
    sink = oal::StatusSink{status + 1, word};
  }
  int rc = forward_entry(p, q, k, v, dim_perm, group_start, packed_coefs(p, factor, factor_rows, kernel_eps, coefs), out, num, den,
                         saved_state, nullptr, workspace, workspace_bytes, status, sink, stream);
  if (ticket) finish_delivery(*ticket, rc, static_cast<cudaStream_t>(stream));
  return rc;
}

int oal_backward(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                 const int32_t* group_start, const float* coef_a, const float* coef_b, const float* coef_c,
                 const float* num, const float* den, const void* saved_state, const void* grad_out,
                 const float* grad_num, const float* grad_den, void* dq, void* dk, void* dv,
                 float* d_coef_a, float* d_coef_b, float* d_coef_c, const float* dstate_in, void* workspace,
                 size_t workspace_bytes, int32_t* status, void* stream) {
  if (int rc = check_problem(p)) return rc;
  if (!q || !k || !v || !dim_perm || !group_start || !coef_a || !coef_b || !coef_c || !num || !den || !status)
    return fail(OAL_ERR_ARGUMENT, "oal_backward: NULL tensor pointer");
  const int mask = p->grad_mask;
  if ((mask & OAL_GRAD_Q) && !dq) return fail(OAL_ERR_ARGUMENT, "dq requested but NULL");
  if ((mask & OAL_GRAD_K) && !dk) return fail(OAL_ERR_ARGUMENT, "dk requested but NULL");
  if ((mask & OAL_GRAD_V) && !dv) return fail(OAL_ERR_ARGUMENT, "dv requested but NULL");
  if ((mask & OAL_GRAD_COEF) && (!d_coef_a || !d_coef_b || !d_coef_c))
    return fail(OAL_ERR_ARGUMENT, "coefficient gradients requested but NULL");
  BackwardArgs x{q, k, v, dim_perm, group_start, num, den, saved_state, grad_out, grad_num, grad_den, dq, dk, dv, dstate_in,
                 workspace, workspace_bytes, status, false};
  return backward_core(p, x, explicit_coefs(coef_a, coef_b, coef_c), CoefSink{d_coef_a, d_coef_b, d_coef_c, nullptr},
                       static_cast<cudaStream_t>(stream));
}

int oal_backward_packed(const OalProblem* p, const void* q, const void* k, const void* v, const int32_t* dim_perm,
                        const int32_t* group_start, const float* factor, int factor_rows, const float* coefs, const float* num,
                        const float* den, const void* saved_state, const void* grad_out, const float* grad_num,
                        const float* grad_den, void* dq, void* dk, void* dv, float* d_factor, void* workspace,
                        size_t workspace_bytes, int32_t* status, int64_t* ticket, void* stream) {
  if (int rc = check_problem(p)) return rc;
  if (!q || !k || !v || !dim_perm || !group_start || !factor || !coefs || !num || !den || !status)
    return fail(OAL_ERR_ARGUMENT, "oal_backward_packed: NULL tensor pointer");
  if (factor_rows != 1 && factor_rows != p->q_heads) return fail(OAL_ERR_ARGUMENT, "oal_backward_packed: factor_rows must be 1 or q_heads");
  const int mask = p->grad_mask;
  if (((mask & OAL_GRAD_Q) && !dq) || ((mask & OAL_GRAD_K) && !dk) || ((mask & OAL_GRAD_V) && !dv) || ((mask & OAL_GRAD_COEF) && !d_factor))
    return fail(OAL_ERR_ARGUMENT, "oal_backward_packed: a requested gradient is NULL");
  oal::StatusSink sink{nullptr, nullptr};
  if (ticket) {
    int32_t* word = nullptr;
    if (int rc = take_delivery(&word, ticket)) return rc;
    sink = oal::StatusSink{nullptr, word};
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BackwardArgs x{q, k, v, dim_perm, group_start, num, den, saved_state, grad_out, grad_num, grad_den, dq, dk, dv, nullptr,
                 workspace, workspace_bytes, status, true};
  CoefSource src = packed_coefs(p, factor, factor_rows, 0.f, const_cast<float*>(coefs));
  int rc = backward_core(p, x, src, CoefSink{nullptr, nullptr, nullptr, (mask & OAL_GRAD_COEF) ? d_factor : nullptr}, st);
  if (!rc && sink.host) {
    LaunchScope scope("deliver_status", st);
    const cudaError_t e = oal::deliver_status(status, sink, st);
    if (e != cudaSuccess) rc = fail_cuda(e, "status delivery kernel");
  }
  if (ticket) finish_delivery(*ticket, rc, st);
  return rc;
}

void oal_set_overlap(int enable) { g_overlap.store(enable ? 1 : 0); }

int oal_status_defer(const int32_t* status, void* stream, int64_t* ticket) {
  if (!status || !ticket) return fail(OAL_ERR_ARGUMENT, "oal_status_defer: NULL pointer");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail_cuda(e, "oal_status_defer");
  if (dev < 0 || dev >= 64) return fail(OAL_ERR_ARGUMENT, "oal_status_defer: device index out of range");
  std::lock_guard<std::mutex> lock(g_status_mutex);
  StatusRing& r = g_status[dev];
  if (!r.stream) {
    if ((e = cudaStreamCreateWithFlags(&r.stream, cudaStreamNonBlocking)) != cudaSuccess) return fail_cuda(e, "oal_status_defer");
    if ((e = cudaHostAlloc(reinterpret_cast<void**>(&r.host), STATUS_RING * sizeof(int32_t), cudaHostAllocPortable)) !=
        cudaSuccess)
      return fail_cuda(e, "oal_status_defer");
  }
  const int slot = (int)(r.next % STATUS_RING);
  if (!r.done[slot]) {
    if ((e = cudaEventCreateWithFlags(&r.ready[slot], cudaEventDisableTiming)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&r.done[slot], cudaEventDisableTiming)) != cudaSuccess)
      return fail_cuda(e, "oal_status_defer");
  } else if ((e = cudaEventSynchronize(r.done[slot])) != cudaSuccess) {   // the slot's previous copy (1024 calls ago)
    return fail_cuda(e, "oal_status_defer");
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if ((e = cudaEventRecord(r.ready[slot], st)) != cudaSuccess || (e = cudaStreamWaitEvent(r.stream, r.ready[slot], 0)) != cudaSuccess ||
      (e = cudaMemcpyAsync(r.host + slot, status, sizeof(int32_t), cudaMemcpyDeviceToHost, r.stream)) != cudaSuccess ||
      (e = cudaEventRecord(r.done[slot], r.stream)) != cudaSuccess)
    return fail_cuda(e, "oal_status_defer");
  *ticket = ((int64_t)dev << 48) | (int64_t)r.next;
  ++r.next;
  return OAL_OK;
}

int oal_status_poll(int64_t ticket, int block, int32_t* value) {
  if (!value) return fail(OAL_ERR_ARGUMENT, "oal_status_poll: NULL pointer");
  if (ticket & TICKET_DELIVERED) return poll_delivery(ticket, block != 0, value);
  const int dev = (int)(ticket >> 48);
  const long long seq = (long long)(ticket & (((int64_t)1 << 48) - 1));
  if (dev < 0 || dev >= 64) return fail(OAL_ERR_ARGUMENT, "oal_status_poll: bad ticket");
  cudaEvent_t done;
  int32_t* word;
  {
    std::lock_guard<std::mutex> lock(g_status_mutex);
    StatusRing& r = g_status[dev];
    if (seq >= r.next || seq + STATUS_RING <= r.next) return fail(OAL_ERR_ARGUMENT, "oal_status_poll: ticket expired or unknown");
    done = r.done[seq % STATUS_RING];
    word = r.host + seq % STATUS_RING;
  }
  if (block) {
    cudaError_t e = cudaEventSynchronize(done);
    if (e != cudaSuccess) return fail_cuda(e, "oal_status_poll");
  } else {
    cudaError_t e = cudaEventQuery(done);
    if (e == cudaErrorNotReady) return 0;
    if (e != cudaSuccess) return fail_cuda(e, "oal_status_poll");
  }
  *value = *static_cast<volatile int32_t*>(word);
  return 1;
}

int oal_expand_factor(const float* factor, int factor_rows, int q_heads, int groups, float kernel_eps, float* coef_a,
                      float* coef_b, float* coef_c, void* stream) {
  if (!factor || !coef_a || !coef_b || !coef_c) return fail(OAL_ERR_ARGUMENT, "oal_expand_factor: NULL pointer");
  if (q_heads < 1 || groups < 1 || groups > OAL_MAX_GROUPS || (factor_rows != 1 && factor_rows != q_heads))
    return fail(OAL_ERR_ARGUMENT, "oal_expand_factor: bad geometry");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  LaunchScope scope("expand_factor", st);
  cudaError_t e = oal::expand_factor(factor, factor_rows, q_heads, groups, kernel_eps, coef_a, coef_b, coef_c, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "oal_expand_factor");
}

int oal_expand_factor_grad(const float* factor, int factor_rows, int q_heads, int groups, const float* d_coef_a,
                           const float* d_coef_b, const float* d_coef_c, float* d_factor, void* stream) {
  if (!factor || !d_coef_a || !d_coef_b || !d_coef_c || !d_factor)
    return fail(OAL_ERR_ARGUMENT, "oal_expand_factor_grad: NULL pointer");
  if (q_heads < 1 || groups < 1 || groups > OAL_MAX_GROUPS || (factor_rows != 1 && factor_rows != q_heads))
    return fail(OAL_ERR_ARGUMENT, "oal_expand_factor_grad: bad geometry");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  LaunchScope scope("expand_factor_grad", st);
  cudaError_t e = oal::expand_factor_grad(factor, factor_rows, q_heads, groups, d_coef_a, d_coef_b, d_coef_c, d_factor, st);
  return e == cudaSuccess ? OAL_OK : fail_cuda(e, "oal_expand_factor_grad");
}

int oal_forward_local_state(const OalProblem* p, const void* k, const void* v, float* state_total, void* workspace,
                            size_t workspace_bytes, int32_t* status, void* stream) {
  int rc = check_problem(p);
  if (rc) return rc;
  if (p->precision != OAL_PRECISION_BF16_TENSORCORE)
    return fail(OAL_ERR_DTYPE, "oal_forward_local_state: chunk states exist only in bf16_tensorcore mode");
  if (!k || !v || !state_total || !status) return fail(OAL_ERR_ARGUMENT, "oal_forward_local_state: NULL tensor pointer");
  if (misaligned({k, v, state_total, workspace})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_forward_local_state");
  ForwardSpaceTC s = carve_forward_tc(p, workspace);
  if (!workspace || workspace_bytes < s.bytes) return fail(OAL_ERR_WORKSPACE, "oal_forward_local_state: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int units = p->batch * p->kv_heads, nb = chunk_count(p);
  cudaError_t e;
  { LaunchScope scope("state_update", st); e = oal::state_update(k, v, s.ds, units, p->seq_len, nb, nb, status, st); }
  if (e != cudaSuccess) return fail_cuda(e, "state update kernel");
  { LaunchScope scope("state_total", st); e = oal::state_scan(s.ds, nullptr, nullptr, nullptr, state_total, units, nb, 0, false, st); }
  if (e != cudaSuccess) return fail_cuda(e, "state total kernel");
  return OAL_OK;
}

int oal_backward_local_state(const OalProblem* p, const void* q, const int32_t* dim_perm, const int32_t* group_start,
                             const float* coef_a, const float* coef_b, const float* coef_c, const float* num,
                             const float* den, const void* saved_state, const void* grad_out, const float* grad_num,
                             const float* grad_den, float* dstate_total, void* workspace, size_t workspace_bytes,
                             int32_t* status, void* stream) {
  int rc = check_problem(p);
  if (rc) return rc;
  if (p->precision != OAL_PRECISION_BF16_TENSORCORE)
    return fail(OAL_ERR_DTYPE, "oal_backward_local_state: chunk states exist only in bf16_tensorcore mode");
  if (p->flags & OAL_FLAG_NO_BACKWARD) return fail(OAL_ERR_ARGUMENT, "oal_backward_local_state: the problem says that no backward follows");
  if (!q || !dim_perm || !group_start || !coef_a || !coef_b || !coef_c || !num || !den || !saved_state || !dstate_total || !status)
    return fail(OAL_ERR_ARGUMENT, "oal_backward_local_state: NULL tensor pointer");
  if (misaligned({q, num, saved_state, grad_out, grad_num, dstate_total, workspace}))
    return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_backward_local_state");
  BackwardSpaceTC s = carve_backward_tc(p, workspace);
  if (!workspace || workspace_bytes < s.bytes) return fail(OAL_ERR_WORKSPACE, "oal_backward_local_state: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  OalProblem local = *p;
  local.grad_mask |= OAL_GRAD_K;      // dCarry is needed whatever the caller finally asks for
  if ((rc = backward_vjp(&local, num, den, grad_out, grad_num, grad_den, s, row_images(&local, saved_state, q, nullptr, nullptr, s.q_image), nullptr, st))) return rc;
  if ((rc = backward_dstate(&local, saved_state, ChunkRange{false, chunk_count(p), 0}, s, status, st))) return rc;
  cudaError_t e;
  { LaunchScope scope("state_total", st);
    e = oal::state_scan(s.dcarry, nullptr, nullptr, nullptr, dstate_total, p->batch * p->kv_heads, chunk_count(p), 1, false, st); }
  if (e != cudaSuccess) return fail_cuda(e, "state gradient total kernel");
  return OAL_OK;
}

// ---------------------------------------------------------------------------------------------
// Forward with library-owned scratch (no caller workspace, no allocation of any kind).
//
// Some hosts of this library cannot obtain device memory at call time: an inference server whose
// memory pool was carved up and frozen at start-up, a plugin that runs inside someone else's
// allocator-free execution callback, a process near its memory limit where cudaMalloc may fail or
// stall.  For them the tensor-core forward keeps its scratch buffer -- the per-chunk
// state increments -- in the file-scope device array below.  The array has
// a fixed size, so the entry point only accepts problems up to kStaticMaxUnitChunks (batch x KV heads
// x 128-token chunks) and kStaticMaxHeads query heads; every GPU that loads the library holds the
// array (about 12.5 MB) until the process exits.
// ---------------------------------------------------------------------------------------------
constexpr int kStaticMaxUnitChunks = 16;
constexpr int kStaticMaxHeads = 64;
constexpr size_t kStaticStateFloats = (size_t)kStaticMaxUnitChunks * OAL_STATE_ROWS * OAL_E_PAD;
static __device__ __align__(256) float g_static_scratch[kStaticStateFloats];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
float* g_static_ptr[kMaxDevices] = {nullptr};

// Device address of g_static_scratch on the current device, resolved once per device.  In host code
// the array's name is only a handle for the runtime, not an address a kernel could use.
int static_scratch_address(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail_cuda(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return fail(OAL_ERR_ARGUMENT, "device ordinal out of range for the static scratch table");
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_ptr[dev]) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_scratch);
    if (e != cudaSuccess) return fail_cuda(e, "cudaGetSymbolAddress(static scratch)");
    g_static_ptr[dev] = ptr;
  }
  *out = g_static_ptr[dev];
  return OAL_OK;
}
}  // namespace

int oal_forward_static_scratch(const OalProblem* p, const void* q, const void* k, const void* v,
                               const int32_t* dim_perm, const int32_t* group_start, const float* coef_a,
                               const float* coef_b, const float* coef_c, void* out, float* num, float* den,
                               void* saved_state, int32_t* status, void* stream) {
  int rc = check_problem(p);
  if (rc) return rc;
  if (p->precision != OAL_PRECISION_BF16_TENSORCORE)
    return fail(OAL_ERR_DTYPE, "oal_forward_static_scratch: only bf16_tensorcore uses scratch memory (fp32_ieee forward needs none: call oal_forward)");
  if (!q || !k || !v || !dim_perm || !group_start || !coef_a || !coef_b || !coef_c || !out || !num || !den || !status || !saved_state)
    return fail(OAL_ERR_ARGUMENT, "oal_forward_static_scratch: NULL tensor pointer");
  if (misaligned({q, k, v, out, num, saved_state})) return fail(OAL_ERR_ARGUMENT, kMisaligned, "oal_forward_static_scratch");
  const int units = p->batch * p->kv_heads, nb = chunk_count(p);
  if ((long long)units * nb > kStaticMaxUnitChunks)
    return fail(OAL_ERR_WORKSPACE, "oal_forward_static_scratch: batch x kv_heads x ceil(seq_len/128) exceeds the static scratch limit of 16; use oal_forward with a caller workspace");
  if (p->q_heads > kStaticMaxHeads)
    return fail(OAL_ERR_WORKSPACE, "oal_forward_static_scratch: more than 64 query heads; use oal_forward with a caller workspace");
  float* scratch = nullptr;
  rc = static_scratch_address(&scratch);
  if (rc) return rc;
  return forward_core(p, q, k, v, dim_perm, group_start, explicit_coefs(coef_a, coef_b, coef_c), out, num, den, saved_state,
                      nullptr, scratch, status, oal::StatusSink{nullptr, nullptr}, false, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
