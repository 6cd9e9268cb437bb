// Runtime state: lazy initialisation, the tensor-format registry, scratch space.
#include "runtime.h"

#include <cstring>

#include "graph_replay.h"
#include "kernels.h"

namespace occ {

static Runtime *g_rt = nullptr;

void set_error(int code, const char *where) {
  Runtime *r = g_rt;
  if (r && r->last_error == 0) r->last_error = code;
  fprintf(stderr, "[occamy_b200] error %d at %s%s%s\n", code, where,
          code > 0 && code < 1000 ? ": " : "",
          code > 0 && code < 1000 ? cudaGetErrorString((cudaError_t)code) : "");
}

Runtime &rt() {
  if (g_rt) return *g_rt;
  Runtime *r = new Runtime();
  g_rt = r;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    // No usable GPU: this library has no CPU path.  Say so and stop.
    fprintf(stderr, "[occamy_b200] fatal: no CUDA device (%s); the runtime has no CPU fallback\n",
            cudaGetErrorString(e));
    exit(-1);
  }
  r->device = dev;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, dev) == cudaSuccess) {
    r->num_sms = prop.multiProcessorCount;
    if (prop.major != 10) {
      fprintf(stderr,
              "[occamy_b200] fatal: device %d is sm_%d%d; this build contains sm_100a code only\n",
              dev, prop.major, prop.minor);
      exit(-1);
    }
  }
  OCC_CUDA(cudaStreamCreateWithFlags(&r->stream, cudaStreamNonBlocking));
  // Mapped host memory: kernels write it only when a bounded wait has run out, and reading it costs no
  // copy (a blocking 4-byte copy behind every result took 18 us of a batch-1 inference).
  OCC_CUDA(cudaHostAlloc((void **)&r->host_err, sizeof(int), cudaHostAllocMapped));
  if (r->host_err) {
    *r->host_err = 0;
    OCC_CUDA(cudaHostGetDevicePointer((void **)&r->dev_err, r->host_err, 0));
  }
  const char *m = getenv("OCCAMY_MATH");
  if (m && (!strcmp(m, "fp32") || !strcmp(m, "0"))) r->mode = MATH_FP32;
  if (m && (!strcmp(m, "bf16") || !strcmp(m, "1"))) r->mode = MATH_BF16;
  if (m && (!strcmp(m, "fp16") || !strcmp(m, "f16") || !strcmp(m, "2"))) r->mode = MATH_F16;
  const char *l = getenv("OCCAMY_LOG");
  r->log = l && *l && strcmp(l, "0");
  const char *c = getenv("OCCAMY_CACHE_WEIGHTS");
  if (c && !strcmp(c, "0")) r->cache_weights = false;
  return *r;
}

void poll_watchdog() {
  Runtime &r = rt();
  volatile int *word = r.host_err;
  if (!word || !*word) return;
  set_error(*word, "kernel watchdog");
  *word = 0;
}

// ---------------------------------------------------------------- registry
void reg_drop_range(void *p, size_t bytes) {
  Runtime &r = rt();
  const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
  auto it = r.recs.lower_bound(lo);
  if (it != r.recs.begin()) {
    auto prev = std::prev(it);
    if (prev->first + prev->second.bytes > lo) it = prev;
  }
  // Handing out [lo, hi) again ends the life of every tensor it touches (the reference
  // zero-fills the range at this point), so their records go, partly covered ones too.
  while (it != r.recs.end() && it->first < hi) it = r.recs.erase(it);
}

void reg_new(void *p, size_t bytes, Fmt fmt) {
  if (!p || bytes == 0) return;
  reg_drop_range(p, bytes);
  TensorRec rec;
  rec.bytes = bytes;
  rec.fmt = fmt;
  rt().recs[(uintptr_t)p] = rec;
}

TensorRec *reg_find(const void *p, uintptr_t *base) {
  Runtime &r = rt();
  const uintptr_t a = (uintptr_t)p;
  auto it = r.recs.upper_bound(a);
  if (it == r.recs.begin()) return nullptr;
  --it;
  if (a >= it->first + it->second.bytes) return nullptr;
  if (base) *base = it->first;
  return &it->second;
}

bool mode_f16() { return rt().mode == MATH_F16; }

static bool is_in_format(const void *p, Fmt want, int64_t n, int64_t c, int64_t h, int64_t w) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  return rec && base == (uintptr_t)p && rec->fmt == want && rec->n == n && rec->c == c &&
         rec->h == h && rec->w == w;
}

bool is_act16(const void *p, int64_t n, int64_t c, int64_t h, int64_t w) {
  return is_in_format(p, mode_f16() ? FMT_F16_NHWC : FMT_BF16_NHWC, n, c, h, w);
}

bool is_parts(const void *p, int64_t n, int64_t c, int64_t h, int64_t w) {
  return is_in_format(p, FMT_PARTS, n, c, h, w);
}

const __nv_bfloat16 *act16_ptr(const void *p) {
  const TensorRec *rec = reg_find(p, nullptr);
  return (const __nv_bfloat16 *)(rec && rec->home ? rec->home : p);
}

static bool home_in_use(const void *h) {
  Runtime &r = rt();
  if (r.home_held && r.home_held(h)) return true;
  for (const auto &kv : r.recs)
    if (kv.second.home == h) return true;
  return false;
}

void free_idle_homes() {
  Runtime &r = rt();
  graph_forget_all();
  OCC_CUDA(cudaStreamSynchronize(r.stream));
  for (size_t i = 0; i < r.homes.size();) {
    if (home_in_use(r.homes[i].ptr)) {
      ++i;
      continue;
    }
    OCC_CUDA(cudaFree(r.homes[i].ptr));
    r.homes.erase(r.homes.begin() + i);
  }
}

cudaError_t device_malloc(void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  graph_free_memory();
  free_idle_homes();
  e = cudaMalloc(p, bytes);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

void *home_acquire(size_t bytes) {
  Runtime &r = rt();
  constexpr size_t MOST = 6;
  Runtime::Home *fit = nullptr, *spare = nullptr;
  for (Runtime::Home &h : r.homes) {
    if (home_in_use(h.ptr)) continue;
    spare = &h;
    if (h.bytes >= bytes && (!fit || h.bytes < fit->bytes)) fit = &h;
  }
  if (fit) return fit->ptr;
  graph_stop_capture();
  if (spare && r.homes.size() >= MOST) {   // too small: replaced
    graph_forget_all();
    OCC_CUDA(cudaStreamSynchronize(r.stream));
    OCC_CUDA(cudaFree(spare->ptr));
    r.homes.erase(r.homes.begin() + (spare - r.homes.data()));
  }
  void *p = nullptr;
  const size_t want = (bytes + 0xFFFFF) & ~(size_t)0xFFFFF;
  OCC_CUDA(device_malloc(&p, want));
  if (p) r.homes.push_back(Runtime::Home{p, want});
  return p;
}

bool is_zero(const void *p) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  return rec && rec->fmt == FMT_ZERO;
}

void mark_f32(void *p) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  if (!rec) return;
  if (base != (uintptr_t)p && rec->fmt != FMT_F32) {
    ensure_f32((const void *)base);  // partial overwrite of a specially formatted tensor
    return;
  }
  rec->fmt = FMT_F32;
  rec->home = rec->dev_src = nullptr;
  rec->host_src = nullptr;
}

static void mark_format(void *p, Fmt fmt, int64_t n, int64_t c, int64_t h, int64_t w, const void *home) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  if (!rec || base != (uintptr_t)p) {
    // Unknown or interior pointer: record it as its own tensor of the fp32 extent.
    reg_new(p, (size_t)(n * c * h * w) * 4, fmt);
    rec = reg_find(p, &base);
  }
  rec->fmt = fmt;
  rec->n = n;
  rec->c = c;
  rec->h = h;
  rec->w = w;
  rec->home = home;
  rec->dev_src = nullptr;
  rec->host_src = nullptr;
}

void mark_act16(void *p, int64_t n, int64_t c, int64_t h, int64_t w, const void *home) {
  mark_format(p, mode_f16() ? FMT_F16_NHWC : FMT_BF16_NHWC, n, c, h, w, home);
}

void mark_parts(void *p, int64_t n, int64_t c, int64_t h, int64_t w, const void *home) {
  mark_format(p, FMT_PARTS, n, c, h, w, home);
}

void ensure_f32(const void *p) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  if (!rec || rec->fmt == FMT_F32) return;
  Runtime &r = rt();
  if (rec->fmt != FMT_ELIDED && r.before_write) {
    const Fmt keep = rec->fmt;
    r.before_write((const void *)base, rec->bytes);
    rec = reg_find(p, &base);          // the hook may have launched work that re-tags tensors
    if (!rec || rec->fmt != keep) return ensure_f32(p);
  }
  if (rec->fmt == FMT_ELIDED) {
    set_error(990, "read of a tensor that cross-call fusion skipped (set OCCAMY_FUSE_ACROSS_CALLS=0)");
  } else if (rec->fmt == FMT_ZERO) {
    enqueue_zero((void *)base, rec->bytes, r.stream);
    r.main_copies++;
  } else if (rec->fmt == FMT_PENDING) {
    graph_stop_capture();
    OCC_CUDA(cudaMemcpyAsync((void *)base, rec->host_src, rec->host_bytes, cudaMemcpyHostToDevice,
                             r.stream));
    r.main_copies++;
    count(CNT_H2D_BYTES, (int64_t)rec->host_bytes);
  } else if (rec->dev_src) {
    graph_stop_capture();   // the caller's memory, elsewhere in the next inference
    enqueue_copy((void *)base, rec->dev_src, (size_t)(rec->n * rec->c * rec->h * rec->w) * 4, r.stream);
    r.main_copies++;
    rec->home = rec->dev_src = nullptr;
  } else if (fmt_is_16(rec->fmt)) {
    const void *tmp = rec->home;
    if (!tmp) {
      const size_t elems = (size_t)(rec->n * rec->c * rec->h * rec->w);
      void *copy = scratch_get(3, elems * 2);
      enqueue_copy(copy, (void *)base, elems * 2, r.stream);
      tmp = copy;
    }
    rec->home = nullptr;
    launch_nhwc_bf16_to_nchw_f32((const bf16 *)tmp, (float *)base, (int)rec->n, (int)rec->c,
                                 (int)rec->h, (int)rec->w, rec->fmt == FMT_F16_NHWC, r.stream);
    count(CNT_MATERIALIZE);
  } else if (rec->fmt == FMT_PARTS) {
    launch_join3_nchw((const bf16 *)rec->home, (float *)base, (int)rec->n, (int)rec->c, (int)rec->h, (int)rec->w,
                      r.stream);
    rec->home = nullptr;
    count(CNT_MATERIALIZE);
  }
  rec->fmt = FMT_F32;
}

void went_forwards() { rt().descending = 1; }

void settle_sources() {
  std::vector<uintptr_t> all;
  for (const auto &kv : rt().recs)
    if (kv.second.dev_src) all.push_back(kv.first);
  for (uintptr_t p : all) ensure_f32((const void *)p);
}

void *scratch_get(int slot, size_t bytes) {
  Runtime &r = rt();
  if (r.scratch_bytes[slot] >= bytes) return r.scratch[slot];
  // Growing: work already enqueued may still use the old block.
  graph_forget_all();
  if (r.scratch[slot]) {
    OCC_CUDA(cudaStreamSynchronize(r.stream));
    OCC_CUDA(cudaFree(r.scratch[slot]));
  }
  size_t want = bytes + bytes / 8;
  want = (want + 0xFFFFF) & ~(size_t)0xFFFFF;
  void *p = nullptr;
  OCC_CUDA(device_malloc(&p, want));
  r.scratch[slot] = p;
  r.scratch_bytes[slot] = p ? want : 0;
  return p;
}

}  // namespace occ
