// Process-wide state of the operator runtime: the launch stream, the registry that
// records in which format each caller-owned tensor currently sits, scratch space,
// the resident packed-weight cache and the error / counter words.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <unordered_map>
#include <vector>

namespace occ {

// Arithmetic of the convolution / GEMM kernels and storage of the activations between them:
// fp32 NCHW throughout; or tensor cores on 16-bit NHWC activations, bf16 (8 mantissa bits, fp32's
// range) or fp16 (11 mantissa bits, values up to 65504).
enum MathMode { MATH_FP32 = 0, MATH_BF16 = 1, MATH_F16 = 2 };

// Format of the bytes behind a caller-owned device pointer.
enum Fmt {
  FMT_F32 = 0,        // what the ABI says: dense fp32, NCHW
  FMT_ZERO = 1,       // freshly handed out; reads as zero, memset not yet issued
  FMT_BF16_NHWC = 2,  // produced by a tensor-core-mode kernel: bf16, NHWC, dims below
  FMT_PENDING = 3,    // host->device upload deferred (constant already packed on device)
  FMT_ELIDED = 4,     // never written: a cross-call fusion skipped it (reading it is an error)
  FMT_F16_NHWC = 5,   // like FMT_BF16_NHWC with fp16 elements (MATH_F16)
  FMT_STEM_ROWS = 6,  // padded channels-last rows for a few-channel convolution, in `home`
  FMT_PARTS = 7       // fp32 as three bf16 parts: three NHWC planes in `home` (fp32 mode, kernels_parts.cu)
};
inline bool fmt_is_16(Fmt f) { return f == FMT_BF16_NHWC || f == FMT_F16_NHWC; }

struct TensorRec {
  size_t bytes = 0;  // extent of the allocation handed to the caller
  Fmt fmt = FMT_F32;
  int64_t n = 0, c = 0, h = 0, w = 0;  // logical NCHW dims of a 16-bit NHWC tensor
  // Where a 16-bit tensor's bytes are when not at the tensor's own address (home_acquire()): its
  // address was still to be read by the kernel that wrote it, or the tensor outlives its address.
  const void *home = nullptr;
  // Caller's device memory the tensor was copied from, when the copy brought it in in another form; the plain
  // form is fetched from there if something asks for it after all, and before the caller can know that the
  // copy has been made and use that memory for something else (settle_sources()).
  const void *dev_src = nullptr;
  int stem_wp = 0, stem_cp = 0, stem_pad = 0, stem_f16 = 0;   // FMT_STEM_ROWS: its geometry and element type
  const void *host_src = nullptr;      // source of the last host->device upload, if any
  size_t host_bytes = 0;
  uint64_t host_hash = 0;
};

struct PackedWeight {
  void *dev = nullptr;
  size_t bytes = 0;
  uint64_t hash = 0;
  int layout = 0;  // packing variant, see pack_weights()
};

struct WeightKey {
  const void *src;
  size_t bytes;
  int layout;
  bool operator==(const WeightKey &o) const {
    return src == o.src && bytes == o.bytes && layout == o.layout;
  }
};
struct WeightKeyHash {
  size_t operator()(const WeightKey &k) const {
    return std::hash<const void *>()(k.src) ^ (k.bytes * 1000003u) ^ (size_t)k.layout * 7919u;
  }
};

enum Counter {
  CNT_LAUNCHES = 0,
  CNT_H2D_BYTES = 1,
  CNT_H2D_SKIPPED = 2,
  CNT_POOL_HWM = 3,
  CNT_TC_LAUNCHES = 4,
  CNT_MATERIALIZE = 5,
  CNT_TMAP_ENCODES = 6,
  CNT_SIMT_LAUNCHES = 7,
  // which forms ran (occamy_get_form_counters)
  CNT_SPLIT_REDUCTION = 8,
  CNT_INVERTED_RESIDUAL = 9,
  CNT_COLUMN_STRIPS = 10,
  CNT_POOLED = 11,
  CNT_REPLAYED = 12,
  CNT_IN_PIECES = 13,
  CNT_SUMMED = 14,
  CNT_PAIRS = 15,
  CNT_ROWS = 16,
  CNT_COUNT = 17
};

struct Runtime {
  cudaStream_t stream = nullptr;
  int device = -1;
  int num_sms = 148;
  MathMode mode = MATH_BF16;
  int last_error = 0;
  int64_t counters[CNT_COUNT] = {};
  int64_t main_copies = 0;  // copies / memsets enqueued on the launch stream (not kernels)
  std::map<uintptr_t, TensorRec> recs;  // keyed by device base pointer
  std::unordered_map<WeightKey, PackedWeight, WeightKeyHash> wcache;
  // host sources whose packed form is resident: source -> (bytes, fingerprint)
  std::unordered_map<const void *, std::pair<size_t, uint64_t>> resident;
  void *scratch[9] = {};
  size_t scratch_bytes[9] = {};
  int *dev_err = nullptr;   // word the kernels' bounded waits report into, as the device sees it
  int *host_err = nullptr;  // the same word (mapped host memory)
  void *host_stage = nullptr;   // pinned, STAGE_BYTES: small results on their way to pageable memory
  bool log = false;
  bool cache_weights = true;
  // The next tensor-core kernel takes its tiles from the last to the first: the one before it took them from the first
  // to the last, and what it wrote last is still in L2 (126 MB, of tensors of 100 to 400 MB).  Kernels that know one
  // order only (went_forwards()) leave it set; the others take turns.  ResNet-50 at 256 images 3287 -> 3221 us, 61
  // at 201x201 938 -> 931, host batches 4531 -> 4493, VGG-16 at 64 1999 -> 1988; small batches the same.
  int descending = 0;
  // called before the runtime itself writes into a caller-owned range (lazy zero fill,
  // deferred upload, layout conversion), so that a held-back kernel can read it first
  void (*before_write)(const void *p, size_t bytes) = nullptr;
  // whether a held-back kernel is still to read the buffer at `home`
  bool (*home_held)(const void *home) = nullptr;
  struct Home {
    void *ptr;
    size_t bytes;
  };
  std::vector<Home> homes;
  // while a piece of a batch is computed by itself (graph_replay.cu): its images and those of the batch
  int64_t piece_images = 0, batch_images = 0;
  // optional CUDA-event pair around every tensor-core launch (occamy_profile_begin/end)
  bool profiling = false;
  int prof_count = 0;
  std::vector<cudaEvent_t> prof_events;
};

// fp32 mode: dense convolutions and GEMMs go to the tensor cores (occamy_set_fp32_tensor_cores)
bool fp32_on_tensor_cores();

Runtime &rt();  // lazily initialised on the current device

// Images that decide in which order a result is summed up: a piece of a batch is computed in the forms (kernel, shares
// of a reduction) that the whole batch takes, so that an image has the same bits either way.
inline int64_t form_images(int64_t n) {
  const Runtime &r = rt();
  return r.piece_images && n == r.piece_images ? r.batch_images : n;
}

void set_error(int code, const char *where);
#define OCC_CUDA(call)                                        \
  do {                                                        \
    cudaError_t e_ = (call);                                  \
    if (e_ != cudaSuccess) ::occ::set_error((int)e_, #call);  \
  } while (0)

constexpr size_t STAGE_BYTES = 256 * 1024;
// After a wait for the stream: report a kernel whose bounded wait ran out, if any.
void poll_watchdog();

// ---- registry --------------------------------------------------------------
// Record that [p, p+bytes) now is a fresh tensor; drops records it overlaps.
void reg_new(void *p, size_t bytes, Fmt fmt);
void reg_drop_range(void *p, size_t bytes);
// Record that contains p, or nullptr.  *base receives its base pointer.
TensorRec *reg_find(const void *p, uintptr_t *base = nullptr);
// Make the bytes behind p plain fp32 NCHW (memset, upload or layout conversion as needed).
void ensure_f32(const void *p);
// The same for every tensor that would have to be fetched from where it was copied from (TensorRec::dev_src).
void settle_sources();
// True when p is the base of a 16-bit NHWC tensor with exactly these logical dims, stored in
// the element type of the CURRENT mode (a tensor left behind in the other 16-bit type is
// converted back to fp32 by its next reader, like any other foreign format).
bool is_act16(const void *p, int64_t n, int64_t c, int64_t h, int64_t w);
// Mark p as fully overwritten by an fp32 kernel / by a 16-bit NHWC kernel of the current mode
// (`home`: into that buffer instead of p's own bytes).
void mark_f32(void *p);
void mark_act16(void *p, int64_t n, int64_t c, int64_t h, int64_t w, const void *home = nullptr);
// The same for fp32 values in three planes (FMT_PARTS); they always have a buffer of their own.
bool is_parts(const void *p, int64_t n, int64_t c, int64_t h, int64_t w);
void mark_parts(void *p, int64_t n, int64_t c, int64_t h, int64_t w, const void *home);
// The bytes of a tensor that is_act16() or is_parts().
const __nv_bfloat16 *act16_ptr(const void *p);
// A buffer for a 16-bit tensor that cannot be written at its own address; in use as long as a tensor
// record (or a kernel that is held back, see home_held) refers to it.  Up to six are kept for the next tensors, more
// while more are in use at a time.
void *home_acquire(size_t bytes);
// The current mode stores fp16 (else bf16) in its 16-bit tensors.
bool mode_f16();
// A tensor that reads as zero and has not been written since it was handed out.
bool is_zero(const void *p);

// cudaMalloc, with a second attempt when the runtime has memory to give back (buffers no tensor is in, what batches in
// pieces work in).
cudaError_t device_malloc(void **p, size_t bytes);
void free_idle_homes();
void *scratch_get(int slot, size_t bytes);
// Error word of the allocation-free entry point on the current device (0 when it was never
// used there); see no_alloc.cu.
int noalloc_poll_error(bool clear);
// Fingerprint of a host buffer; of one up to HASH_WHOLE bytes every byte counts, of a larger one a sample.
constexpr size_t HASH_WHOLE = 16 * 1024;
uint64_t host_hash(const void *src, size_t bytes);

inline void count(Counter c, int64_t v = 1) { rt().counters[c] += v; }
inline int64_t numel4(const int64_t *d) { return d[0] * d[1] * d[2] * d[3]; }

}  // namespace occ
