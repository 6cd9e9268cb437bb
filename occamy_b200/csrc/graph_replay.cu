// Capture, matching and launch of recorded inferences (see graph_replay.h).
#include "graph_replay.h"

#include <cstring>
#include <map>

#include "kernels.h"

namespace occ {

#ifdef OCCAMY_TUNING
#define GR_LOG(...) do { if (getenv("OCCAMY_GRAPH_LOG")) fprintf(stderr, "[graph] " __VA_ARGS__); } while (0)
#else
#define GR_LOG(...) do {} while (0)
#endif

namespace {

// First graph of an inference: few kernels, so that the GPU starts while the host still checks
// calls (and fingerprints constants) of the rest.
constexpr int64_t FIRST_GRAPH_LAUNCHES = 12;
constexpr size_t MAX_VARIANTS = 8;   // per program: pool blocks x sets of constants x modes
constexpr int MAX_FAILURES = 3;      // captures broken off before a program is left alone

struct SavedRec {
  size_t offset;   // in the pool
  TensorRec rec;
};

// A window cut up by images: its calls are made for a piece of the batch after the other, each piece as one
// graph, on tensors in memory of the runtime's.  What it is for is a batch that comes from the host: the
// pieces are computed while the later ones are still on their way (batch 256 of a ResNet-50 takes 2.8 ms to
// arrive and 2.6 to compute).
constexpr int MAX_PIECES = 4;

// An executable graph.  One that goes out of use may still be running: it is destroyed later (empty_trash()).
struct Exec {
  cudaGraphExec_t e = nullptr;
  Exec() {}
  Exec(Exec &&o) : e(o.e) { o.e = nullptr; }
  Exec &operator=(Exec &&o) {
    std::swap(e, o.e);
    return *this;
  }
  ~Exec();
};

struct Segment {
  Exec exec;                        // null: the calls enqueue nothing
  Exec pieces[MAX_PIECES];          // instead of exec, in a window cut up by images
  size_t end = 0;                   // one past its last call
  std::vector<SavedRec> after;      // registry records of the pool when it has been enqueued
  int64_t counters[CNT_COUNT] = {};   // what its calls count
  int64_t copies = 0, chains = 0;
};

struct Constant {
  size_t call;
  const void *src;
  uint64_t hash;
};

// What the last graph of a window cut up by images moves: the result to its tensor; and what was there of the
// batch, which is still needed should the window have to be made call by call after all, out of the way.
struct ResultCopy {
  void *tensor = nullptr, *made = nullptr, *aside = nullptr;
  size_t bytes = 0;
};

struct Variant {
  uintptr_t pool_base = 0;
  int flags = 0;
  uint64_t epoch = 0, used = 0;
  std::vector<SavedRec> before;   // the pool's records when the window began: the forms its inputs are in
  std::vector<Constant> constants;
  std::vector<Segment> segments;
  bool pieces = false;            // one segment, cut up by images
  ResultCopy result;
};

}  // namespace

struct GraphPlan {
  size_t begin = 0, end = 0;   // the window: calls [begin, end)
  bool ready = false;          // an inference ran with nothing to upload or allocate inside it
  int failures = 0;
  int piece_failures = 0;
  std::vector<std::unique_ptr<Variant>> variants;
};

namespace {

enum State { IDLE, CAPTURING, REPLAYING, PLAIN };   // PLAIN: this inference runs call by call

struct Replay {
  State state = PLAIN;
  TraceProgram *prog = nullptr;
  bool again = false;                 // run_again() is making calls
  uint64_t epoch = 1, tick = 0;
  uint64_t epoch_at_begin = 0;
  bool disturbed = false;             // this inference allocated, uploaded or waited inside its calls
  // replaying
  size_t next = 0;                    // call expected next
  size_t seg = 0;                     // segment it belongs to
  std::vector<Variant *> left;        // variants that agree so far; the first one is launched
  size_t constant = 0;                // constants checked so far
  std::vector<const void *> hosts;    // sources of this inference's constants, per call of the window
  // capturing
  std::unique_ptr<Variant> building;
  int64_t base_counters[CNT_COUNT] = {};
  int64_t base_copies = 0, base_chains = 0;
  std::vector<cudaGraphExec_t> trash;   // launched once, destroyed when the stream is idle
  // an upload that is being made in pieces, and the event behind each
  int pieces_coming = 0;
  cudaEvent_t piece_here[MAX_PIECES] = {};
  void *piece_memory = nullptr;         // where the tensors of a window cut up by images are
  size_t piece_bytes = 0;
  bool making_pieces = false;           // build_pieces() is using it
  // this inference ran its window as pieces
  TraceProgram *in_pieces = nullptr;
  const Variant *pieces_of = nullptr;
};
Replay &gr = *new Replay;   // never destroyed, like the programs it refers to

Exec::~Exec() {
  if (e) gr.trash.push_back(e);
}

bool computes(int sym) { return sym >= S_CONV && sym <= S_RESHAPE; }

int mode_flags() {
  const Runtime &r = rt();
  return (int)r.mode * 4 + (r.cache_weights ? 2 : 0) + (fp32_on_tensor_cores() ? 1 : 0);
}

bool allowed() {
  const Runtime &r = rt();
  return !r.profiling && !r.log && r.cache_weights && trace_active();
}

void empty_trash(bool wait) {
  if (gr.trash.empty()) return;
  if (!wait && cudaStreamQuery(rt().stream) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (wait) OCC_CUDA(cudaStreamSynchronize(rt().stream));
  for (cudaGraphExec_t e : gr.trash) cudaGraphExecDestroy(e);
  gr.trash.clear();
}

void save_registry(std::vector<SavedRec> &out, uintptr_t base, size_t bytes) {
  out.clear();
  auto &recs = rt().recs;
  for (auto it = recs.lower_bound(base); it != recs.end() && it->first < base + bytes; ++it)
    out.push_back(SavedRec{it->first - base, it->second});
}

void restore_registry(const std::vector<SavedRec> &in, uintptr_t base, size_t bytes) {
  auto &recs = rt().recs;
  std::map<uintptr_t, const void *> sources;   // this inference's, not those of the captured one
  for (auto it = recs.lower_bound(base); it != recs.end() && it->first < base + bytes; ++it)
    if (it->second.dev_src) sources[it->first] = it->second.dev_src;
  recs.erase(recs.lower_bound(base), recs.lower_bound(base + bytes));
  for (const SavedRec &s : in) {
    TensorRec rec = s.rec;
    if (rec.dev_src) rec.dev_src = sources.count(base + s.offset) ? sources[base + s.offset] : nullptr;
    recs.emplace(base + s.offset, rec);
  }
}

// The same tensors in the same form.  Constants uploaded before the window are among them: the graphs refer to
// what was packed from that very source (of others it does not matter where their contents came from).
bool same_record(const TensorRec &a, const TensorRec &b) {
  if (a.bytes != b.bytes || a.fmt != b.fmt || a.home != b.home) return false;
  if (a.fmt == FMT_PENDING) return a.host_src == b.host_src && a.host_bytes == b.host_bytes && a.host_hash == b.host_hash;
  if (a.fmt == FMT_F32 || a.fmt == FMT_ZERO || a.fmt == FMT_ELIDED) return true;
  return a.n == b.n && a.c == b.c && a.h == b.h && a.w == b.w &&
         (a.fmt != FMT_STEM_ROWS || (a.stem_wp == b.stem_wp && a.stem_cp == b.stem_cp && a.stem_pad == b.stem_pad &&
                                     a.stem_f16 == b.stem_f16));
}

bool same_registry(const std::vector<SavedRec> &a, uintptr_t base, size_t bytes) {
  auto &recs = rt().recs;
  auto it = recs.lower_bound(base);
  for (const SavedRec &s : a) {
    if (it == recs.end() || it->first != base + s.offset || !same_record(it->second, s.rec)) return false;
    ++it;
  }
  return it == recs.end() || it->first >= base + bytes;
}

// ---- recording ------------------------------------------------------------------
// The graph is put together node by node from the runtime's own launches.  (A stream capture would do it too, but
// while a stream of a device captures, any thread's wait for the device fails and makes the capture invalid.)
struct Work {   // one node, enough to enqueue it by itself
  cudaGraphNode_t node;
  void *dst;             // copies and zero fills; null: a kernel
  const void *src;       // null: a zero fill
  size_t bytes;
};
struct Recording {
  cudaGraph_t graph = nullptr;
  std::vector<Work> work;
};
Recording *recording = nullptr;
bool spoiled = false;   // a piece's recording met work that has to be done at once, and was dropped

bool record_begin() {
  std::unique_ptr<Recording> rec(new Recording);
  if (cudaGraphCreate(&rec->graph, 0) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  recording = rec.release();
  return true;
}

// Appends `w`, whose node has no dependencies yet, behind the last one.
bool record_append(const Work &w, bool chained) {
  cudaError_t e = cudaSuccess;
  if (!recording->work.empty()) {
    const Work &last = recording->work.back();
    cudaGraphEdgeData edge = {};
    if (chained && !last.dst) {   // may start while the kernel before it is still running
      edge.from_port = cudaGraphKernelNodePortProgrammatic;
      edge.type = cudaGraphDependencyTypeProgrammatic;
    }
    e = cudaGraphAddDependencies_v2(recording->graph, &last.node, &w.node, &edge, 1);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    cudaGraphDestroyNode(w.node);
    return false;
  }
  recording->work.push_back(w);
  return true;
}

bool record_kernel(const void *kernel, const cudaLaunchConfig_t &cfg, void **args) {
  cudaKernelNodeParams p = {};
  p.func = const_cast<void *>(kernel);
  p.gridDim = cfg.gridDim;
  p.blockDim = cfg.blockDim;
  p.sharedMemBytes = (unsigned)cfg.dynamicSmemBytes;
  p.kernelParams = args;
  Work w = {};
  bool chained = false;
  cudaError_t e = cudaGraphAddKernelNode(&w.node, recording->graph, nullptr, 0, &p);
  for (unsigned i = 0; i < cfg.numAttrs && e == cudaSuccess; ++i) {
    if (cfg.attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization) chained = true;
    else e = cudaGraphKernelNodeSetAttribute(w.node, cfg.attrs[i].id, &cfg.attrs[i].val);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return record_append(w, chained);
}

bool record_copy(void *dst, const void *src, size_t bytes) {
  Work w = {};
  w.dst = dst;
  w.src = src;
  w.bytes = bytes;
  cudaError_t e;
  if (src) {
    e = cudaGraphAddMemcpyNode1D(&w.node, recording->graph, nullptr, 0, dst, src, bytes, cudaMemcpyDeviceToDevice);
  } else {
    cudaMemsetParams m = {};
    m.dst = dst;
    m.elementSize = 1;
    m.width = bytes;
    m.height = 1;
    e = cudaGraphAddMemsetNode(&w.node, recording->graph, nullptr, 0, &m);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return record_append(w, false);
}

// Enqueues the recorded work piece by piece.
void run_recorded(const Recording &rec) {
  const cudaStream_t s = rt().stream;
  for (const Work &w : rec.work) {
    if (w.dst && w.src) {
      OCC_CUDA(cudaMemcpyAsync(w.dst, w.src, w.bytes, cudaMemcpyDeviceToDevice, s));
    } else if (w.dst) {
      OCC_CUDA(cudaMemsetAsync(w.dst, 0, w.bytes, s));
    } else {
      cudaKernelNodeParams p = {};
      cudaLaunchAttribute cluster = {};
      cluster.id = cudaLaunchAttributeClusterDimension;
      OCC_CUDA(cudaGraphKernelNodeGetParams(w.node, &p));
      OCC_CUDA(cudaGraphKernelNodeGetAttribute(w.node, cluster.id, &cluster.val));
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = p.gridDim;
      cfg.blockDim = p.blockDim;
      cfg.dynamicSmemBytes = p.sharedMemBytes;
      cfg.stream = s;
      cfg.attrs = &cluster;
      cfg.numAttrs = cluster.val.clusterDim.x > 1 ? 1 : 0;
      OCC_CUDA(cudaLaunchKernelExC(&cfg, p.func, p.kernelParams));
    }
  }
}

// Ends the recording.  The executable graph, or null when it is empty; false when there is none for another reason.
// With `enqueue` what was recorded is enqueued, either way.
bool record_end(cudaGraphExec_t *exec, bool enqueue) {
  std::unique_ptr<Recording> rec(recording);
  recording = nullptr;
  *exec = nullptr;
  bool ok = true;
  if (!rec->work.empty()) {
    ok = cudaGraphInstantiate(exec, rec->graph, 0) == cudaSuccess &&
         (!enqueue || cudaGraphLaunch(*exec, rt().stream) == cudaSuccess);
    if (!ok) {
      cudaGetLastError();
      if (*exec) cudaGraphExecDestroy(*exec);
      *exec = nullptr;
      if (enqueue) run_recorded(*rec);
    }
  }
  cudaGraphDestroy(rec->graph);
  return ok;
}

bool begin_segment() {
  Runtime &r = rt();
  memcpy(gr.base_counters, r.counters, sizeof(gr.base_counters));
  gr.base_copies = r.main_copies;
  gr.base_chains = trace_fused_chains();
  if (!record_begin()) return false;
  gr.state = CAPTURING;
  return true;
}

bool end_segment(cudaGraphExec_t *exec) {
  gr.state = PLAIN;
  return record_end(exec, true);
}

void add_variant(GraphPlan &plan, std::unique_ptr<Variant> v) {
  auto &vs = plan.variants;
  for (size_t i = 0; i < vs.size();)
    if (vs[i]->epoch != gr.epoch) vs.erase(vs.begin() + i);
    else ++i;
  if (vs.size() >= MAX_VARIANTS) {
    size_t oldest = 0;
    for (size_t i = 1; i < vs.size(); ++i)
      if (vs[i]->used < vs[oldest]->used) oldest = i;
    vs.erase(vs.begin() + oldest);
  }
  vs.push_back(std::move(v));
}

// The calls of the current capture have all been made: keep it.
void close_segment(GraphPlan &plan) {
  Runtime &r = rt();
  Segment s;
  s.end = trace_index();
  const bool last = s.end == plan.end;
  if (last) flush_held_back();
  if (gr.state != CAPTURING) return;   // what was held back needed a new buffer: the capture is broken off
  for (int i = 0; i < CNT_COUNT; ++i) s.counters[i] = r.counters[i] - gr.base_counters[i];
  s.counters[CNT_H2D_SKIPPED] = s.counters[CNT_POOL_HWM] = 0;   // counted as the calls are checked
  s.copies = r.main_copies - gr.base_copies;
  s.chains = trace_fused_chains() - gr.base_chains;
  save_registry(s.after, trace_pool_base(), trace_pool_bytes());
  if (!end_segment(&s.exec.e)) {
    plan.failures = MAX_FAILURES;
    gr.building.reset();
    return;
  }
  gr.building->segments.push_back(std::move(s));
  if (!last) {
    if (!begin_segment()) gr.building.reset();
    return;
  }
  // the fingerprints are those of the calls just made
  const auto &calls = trace_entries();
  for (size_t i = plan.begin; i < plan.end; ++i)
    if (calls[i].sym == S_H2D) {
      gr.building->constants.push_back(Constant{i, calls[i].host, (uint64_t)calls[i].args.v[1]});
    }
  gr.building->used = ++gr.tick;
  add_variant(plan, std::move(gr.building));
}

// ---- after an ordinary inference: is there a window, and was it quiet? ------------------
bool in_pool(uintptr_t p, const TraceProgram &t) {
  return p == 0 || (p >= t.pool_base && p < t.pool_base + t.pool_bytes);
}

void look_for_window(const std::vector<Entry> &calls, TraceProgram &p) {
  if (!p.pool_base || calls.size() != p.entries.size()) return;
  size_t first_compute = calls.size();
  for (size_t i = 0; i < calls.size() && first_compute == calls.size(); ++i)
    if (computes(calls[i].sym)) first_compute = i;
  size_t begin = 0;
  for (size_t i = 0; i < first_compute; ++i) {
    const int s = calls[i].sym;
    const bool quiet = s == S_MEMOFFSET || (s == S_H2D && !calls[i].uploaded);
    if (!quiet) begin = i + 1;
  }
  size_t end = begin;
  for (size_t i = begin; i < calls.size(); ++i) {
    const Entry &e = calls[i];
    const Entry &rec = p.entries[i];
    if (computes(e.sym)) {
      if (!e.args.whole) break;   // could not be made again
      if (!in_pool(rec.in[0], p) || !in_pool(rec.in[1], p) || !in_pool(rec.in[2], p) || !in_pool(rec.out, p)) break;
      end = i + 1;
    } else if (!(e.sym == S_MEMOFFSET || (e.sym == S_H2D && !e.uploaded))) {
      break;
    }
  }
  GR_LOG("window %zu..%zu of %zu\n", begin, end, calls.size());
  if (end == begin) return;
  if (!p.graph) p.graph = std::make_shared<GraphPlan>();
  if (p.graph->begin != begin || p.graph->end != end) p.graph->variants.clear();
  p.graph->begin = begin;
  p.graph->end = end;
  p.graph->ready = true;
}

// ---- replay -----------------------------------------------------------------------
// Takes the inference back to the end of the last launched graph and makes the calls since then.
void take_back() {
  TraceProgram *p = gr.prog;
  GR_LOG("taken back at call %zu (sym %d)\n", gr.next, p->entries[gr.next].sym);
  const Variant &v = *gr.left[0];
  const size_t from = gr.seg ? v.segments[gr.seg - 1].end : p->graph->begin;
  const size_t upto = gr.next;
  const uintptr_t base = trace_pool_base();
  const size_t bytes = trace_pool_bytes();
  if (gr.seg) restore_registry(v.segments[gr.seg - 1].after, base, bytes);
  gr.state = PLAIN;
  gr.left.clear();
  trace_rewind(p, from);
  gr.again = true;
  for (size_t i = from; i < upto; ++i)
    run_again(p->entries[i],
              [&](void *q) {
                const uintptr_t a = (uintptr_t)q;
                return (void *)(a >= p->pool_base && a < p->pool_base + p->pool_bytes ? a - p->pool_base + base : a);
              },
              gr.hosts[i - p->graph->begin]);
  gr.again = false;
}

void wait_for_upload() {
  if (!gr.pieces_coming) return;
  OCC_CUDA(cudaStreamWaitEvent(rt().stream, gr.piece_here[gr.pieces_coming - 1], 0));
  gr.pieces_coming = 0;
}

// ---- windows cut up by images -------------------------------------------------------
// Images of each piece.  The first has to arrive before anything is computed and the last is computed when nothing
// arrives any more; the others cost a start of fifty kernels each.  None is larger than the last (lay_out() makes room for
// that one).  None for batches below 128, nor in the fp32 mode, which computes for longer than the upload takes.
// Milliseconds per inference from pinned memory to host memory, 224x224: whole batch, 1/4 + 3/8 + 3/8, and 3/16 + 1/4 +
// 9/32 + 9/32.
//     images               128                  160                  192                  224                  256
//     ResNet-50    2.89 / 2.36 / 2.47   3.47 / 2.73 / 2.77   4.10 / 3.12 / 3.14   4.78 / 3.55 / 3.51   5.32 / 3.98 / 3.81
//     MobileNetV2  2.32 / 1.99 / 1.96                        3.36 / 2.77 / 2.76                        4.36 / 3.63 / 3.49
//     VGG-16       4.34 / 3.69 / 3.67
// (Below 128, and in the fp32 mode, with the kernels of an earlier build: ResNet-50 with 64 images 1.87 whole and 2.12 in
// pieces, 96 2.50 and 2.53; MobileNetV2 1.38 / 1.30 and 1.89 / 1.67; VGG-16 with 64 2.64 / 2.43; fp32 5.72 / 6.44, 128
// 10.44 / 10.67.)
// The first inference on newly pinned memory takes 1.2 ms longer with 256 images, whole or in pieces: its upload does (a
// copy by itself 4.7 ms there and 3.6 from then on).
int piece_images(int64_t n, int64_t *images) {
  if (n < 128 || rt().mode == MATH_FP32) return 0;
  const int pieces = n < 208 ? 3 : 4;
  images[0] = n / (pieces == 3 ? 8 : 16) * (pieces == 3 ? 2 : 3) / 8 * 8;
  int64_t left = n - images[0];
  if (pieces == 4) left -= images[1] = n / 4 / 8 * 8;
  images[pieces - 2] = left / 2 / 8 * 8;
  images[pieces - 1] = left - images[pieces - 2];
  return pieces;
}

struct Cut {
  std::vector<Entry> calls;    // of the whole inference, those of the window for one piece
  uintptr_t x = 0, out = 0;
  int64_t x_bytes = 0, out_bytes = 0, batch = 0;
  size_t x_until = 0, out_from = 0;   // calls between which these addresses mean the input and the result
  std::vector<size_t> offset;         // of the tensor that a call of the window hands out, in the pieces' memory
  size_t bytes = 0;                   // what these tensors need
};

// Whether the tensor handed out by call `i` is a constant: the first call that writes it is an upload.
bool is_constant(const std::vector<Entry> &calls, size_t i, size_t end) {
  const uintptr_t a = calls[i].out;
  for (size_t j = i + 1; j < end; ++j) {
    if (calls[j].sym == S_H2D && calls[j].out == a) return true;
    if (calls[j].out == a) return false;
  }
  return false;
}

// Places for the window's tensors, as large as a piece needs them: first fit, a tensor's place is free again when the
// pool hands out what it had there.
void lay_out(const TraceProgram &p, Cut &c) {
  struct Live {
    uintptr_t pool;
    int64_t pool_bytes;
    size_t at, bytes;
  };
  std::vector<Live> live;   // by place
  c.offset.assign(p.graph->end - p.graph->begin, 0);
  c.bytes = 0;
  for (size_t i = p.graph->begin; i < p.graph->end; ++i) {
    const Entry &e = p.entries[i];
    if (e.sym != S_MEMOFFSET) continue;
    for (size_t k = 0; k < live.size();)
      if (live[k].pool < e.out + (uintptr_t)e.out_bytes && e.out < live[k].pool + (uintptr_t)live[k].pool_bytes)
        live.erase(live.begin() + k);
      else ++k;
    if (i == c.out_from) continue;
    const size_t bytes = ((size_t)c.calls[i].out_bytes + 255) & ~(size_t)255;
    size_t at = 0, k = 0;
    for (; k < live.size() && live[k].at < at + bytes; ++k) at = live[k].at + live[k].bytes;
    live.insert(live.begin() + k, Live{e.out, e.out_bytes, at, bytes});
    c.offset[i - p.graph->begin] = at;
    if (c.bytes < at + bytes) c.bytes = at + bytes;
  }
}

// The call that uploads the batch: the one right before the window.
bool find_input(const TraceProgram &p, Cut &c) {
  const size_t begin = p.graph->begin;
  if (begin == 0 || p.entries[begin - 1].sym != S_H2D) return false;
  const Entry &up = p.entries[begin - 1];
  c.x = up.out;
  c.x_bytes = up.out_bytes;
  for (size_t i = begin; i < p.graph->end; ++i) {
    const Entry &e = p.entries[i];
    if (e.sym != S_CONV && e.sym != S_CONV_BIAS_ACT) continue;
    c.batch = e.args.v[0];
    return e.in[0] == c.x && e.in_bytes[0] == c.x_bytes;
  }
  return false;
}

// Rewrites the window's calls for `images` of the batch; false when a call is not one image after the other.
bool cut_up(const TraceProgram &p, int64_t images, Cut &c) {
  const int64_t N = c.batch;
  const size_t begin = p.graph->begin, end = p.graph->end;
  std::map<uintptr_t, int64_t> batch, constants;   // tensors by address, with their bytes
  batch[c.x] = c.x_bytes;
  c.x_until = end;
  c.calls = p.entries;
  auto drop = [](std::map<uintptr_t, int64_t> &m, uintptr_t a, int64_t bytes) {
    for (auto it = m.begin(); it != m.end();)
      if (it->first < a + (uintptr_t)bytes && a < it->first + (uintptr_t)it->second) it = m.erase(it);
      else ++it;
  };
  std::map<uintptr_t, size_t> handed_out;   // last call that did
  for (size_t i = 0; i < end; ++i) {
    Entry &e = c.calls[i];
    int64_t *v = e.args.v;
    if (e.sym == S_MEMOFFSET) {
      drop(batch, e.out, e.out_bytes);
      drop(constants, e.out, e.out_bytes);
      handed_out[e.out] = i;
      if (i >= begin && c.x_until == end && !batch.count(c.x)) c.x_until = i;
      if (i < begin && e.out == c.x) batch[c.x] = c.x_bytes;
      if (i >= begin && !is_constant(p.entries, i, end)) {
        e.out_bytes = ((e.out_bytes * images + N - 1) / N + 31) / 32 * 32;
        v[0] = e.out_bytes;
      }
      continue;
    }
    if (e.sym == S_H2D) {
      if (i >= begin) {   // (one that is there before the batch is not the pieces' own)
        if (!handed_out.count(e.out) || handed_out[e.out] < begin) return false;
        constants[e.out] = e.out_bytes;
      }
      continue;
    }
    if (i < begin) continue;
    auto scaled = [&](int64_t &d) {
      if (d != N) return false;
      d = images;
      return true;
    };
    if (!batch.count(e.in[0])) return false;
    if (!handed_out.count(e.out) || handed_out[e.out] < begin) return false;   // (the batch stays as it is)
    bool ok = true, second_scaled = false;
    switch (e.sym) {
      case S_CONV:
      case S_CONV_BIAS_ACT:
        ok = scaled(v[0]) && constants.count(e.in[1]) && (!e.in[2] || constants.count(e.in[2]));
        break;
      case S_ACTIVE: ok = scaled(v[0]); break;
      case S_CLIP: ok = scaled(v[1]); break;
      case S_TENSOR_OP:
        ok = scaled(v[3]);
        if (e.in[1] && batch.count(e.in[1])) ok = ok && v[1] == v[2] && scaled(v[3 + v[1]]) && (second_scaled = true);
        else ok = ok && (!e.in[1] || (constants.count(e.in[1]) && (v[2] < v[1] || v[3 + v[1]] == 1)));
        break;
      case S_MAXPOOL:
      case S_AVGPOOL: ok = scaled(v[0]) && scaled(v[4]); break;
      case S_REDUCE: ok = scaled(v[2]) && scaled(v[2 + v[0]]); break;
      case S_MATMUL: ok = v[4] == 0 && scaled(v[0]) && constants.count(e.in[1]); break;
      case S_SOFTMAX: ok = scaled(v[2]) && v[0] > 0; break;
      case S_FLATTEN:
      case S_RESHAPE: ok = scaled(v[1]); break;
      default: ok = false;
    }
    if (!ok || e.out_bytes % N || e.in_bytes[0] % N) return false;
    batch[e.out] = e.out_bytes;
    if (e.dims[0] == N) e.dims[0] = images;
    e.out_bytes = e.out_bytes / N * images;
    e.in_bytes[0] = e.in_bytes[0] / N * images;
    if (second_scaled) e.in_bytes[1] = e.in_bytes[1] / N * images;
    if (e.sym == S_MATMUL && e.in[2]) e.in_bytes[2] = e.out_bytes;
  }
  // behind the window one tensor is read, rows of fp32, and nothing else happens (graph_left_recording())
  for (size_t i = end; i < c.calls.size(); ++i) {
    const Entry &e = c.calls[i];
    const bool to_pool = e.out >= p.pool_base && e.out < p.pool_base + p.pool_bytes;
    if (e.sym != S_D2H && e.sym != S_POOLFREE && !(e.sym == S_D2D && !to_pool)) return false;
    for (int k = 0; k < 3; ++k) {
      if (!e.in[k] || e.in[k] < p.pool_base || e.in[k] >= p.pool_base + p.pool_bytes) continue;
      if ((c.out && e.in[k] != c.out) || !batch.count(e.in[k]) || e.in_bytes[k] != batch[e.in[k]]) return false;
      c.out = e.in[k];
      c.out_bytes = e.in_bytes[k];
    }
  }
  if (!c.out || !handed_out.count(c.out) || handed_out[c.out] < begin) return false;
  c.out_from = handed_out[c.out];
  for (size_t i = end; i-- > begin;)
    if (c.calls[i].out == c.out && computes(c.calls[i].sym)) {
      const int sym = c.calls[i].sym;
      if (sym != S_MATMUL && sym != S_SOFTMAX && !(sym == S_TENSOR_OP && c.calls[i].kind == CK_ROW_BIAS)) return false;
      break;
    }
  return true;
}

// Makes the window's calls for one piece: images [at, at + images) of the batch.
void make_piece(const TraceProgram &p, const Cut &c, int64_t at, int64_t images, const std::vector<const void *> &hosts) {
  Runtime &r = rt();
  r.piece_images = images;
  r.batch_images = c.batch;
  const uintptr_t real = trace_pool_base(), mine = (uintptr_t)gr.piece_memory;
  std::map<uintptr_t, uintptr_t> where;   // of the window's tensors, by their addresses in the pool
  const uintptr_t x = c.x - p.pool_base + real + (uintptr_t)(c.x_bytes / c.batch * at);
  const uintptr_t out = mine + c.bytes + (uintptr_t)(c.out_bytes / c.batch * at);
  gr.again = true;
  for (size_t i = p.graph->begin; i < p.graph->end; ++i) {
    if (i == c.out_from) {
      reg_new((void *)out, (size_t)(c.out_bytes / c.batch * images), FMT_ZERO);
      continue;
    }
    if (c.calls[i].sym == S_MEMOFFSET) where[c.calls[i].out] = mine + c.offset[i - p.graph->begin];
    trace_force(p.roles[i]);
    run_again(c.calls[i],
              [&](void *q) -> void * {
                const uintptr_t a = (uintptr_t)q;
                if (a < p.pool_base || a >= p.pool_base + p.pool_bytes) return q;
                if (a == c.x && i < c.x_until) return (void *)x;
                if (a == c.out && i > c.out_from) return (void *)out;
                return (void *)where[a];
              },
              hosts[i - p.graph->begin]);
  }
  trace_force_end();
  flush_held_back();
  gr.again = false;
  r.piece_images = r.batch_images = 0;
}

// An inference has just run its window as the graphs of `v`: make the variant that is cut up by images.
void build_pieces(TraceProgram &p, const Variant &v) {
  GraphPlan &plan = *p.graph;
  Cut c;
  int64_t images[MAX_PIECES];
  if (plan.piece_failures >= MAX_FAILURES) return;
  for (const auto &o : plan.variants)
    if (o->pieces && o->pool_base == v.pool_base && o->flags == v.flags && o->epoch == gr.epoch) return;
  const int pieces = find_input(p, c) && c.x_bytes >= (16 << 20) ? piece_images(c.batch, images) : 0;
  if (!pieces || !cut_up(p, images[pieces - 1], c)) {
    plan.piece_failures = MAX_FAILURES;
    return;
  }
  Runtime &r = rt();
  plan.piece_failures++;   // taken back below
  lay_out(p, c);   // for the largest piece; the result of all of them behind it
  const size_t result_room = ((size_t)c.out_bytes + 255) & ~(size_t)255, bytes = c.bytes + 2 * result_room;
  if (gr.piece_bytes < bytes) {
    graph_free_memory();
    if (cudaMalloc(&gr.piece_memory, bytes) != cudaSuccess) {
      cudaGetLastError();
      gr.piece_memory = nullptr;
      plan.piece_failures = MAX_FAILURES;
      return;
    }
    gr.piece_bytes = bytes;
  }
  gr.making_pieces = true;
  const uintptr_t mine = (uintptr_t)gr.piece_memory;
  const std::vector<const void *> hosts = gr.hosts;
  int64_t counters[CNT_COUNT];
  memcpy(counters, r.counters, sizeof(counters));
  const int64_t copies = r.main_copies;
  auto fresh = [&]() { reg_drop_range((void *)mine, gr.piece_bytes); };
  // the batch's own record covers its place, as it will when the window begins
  restore_registry(v.before, v.pool_base, trace_pool_bytes());
  std::unique_ptr<Variant> n(new Variant);
  n->pool_base = v.pool_base;
  n->flags = v.flags;
  n->before = v.before;
  n->constants = v.constants;
  n->pieces = true;
  n->segments.resize(1);
  n->result.tensor = (void *)(c.out - p.pool_base + v.pool_base);
  n->result.made = (void *)(mine + c.bytes);
  n->result.aside = (void *)(mine + c.bytes + result_room);
  n->result.bytes = (size_t)c.out_bytes;
  Segment &s = n->segments[0];
  s.end = plan.end;
  bool ok = true;
  const uint64_t epoch = gr.epoch;
  int64_t at = 0;
  for (int k = 0; k < pieces && ok; at += images[k++]) {
    Cut piece = c;
    piece.out = 0;
    ok = cut_up(p, images[k], piece);
    int64_t copies0 = 0, chains0 = 0;
    // A piece may take kernels, and with them packed constants and buffers, that neither the whole batch nor
    // another piece takes.  Packing and allocating are done, not recorded: they end the recording, what follows
    // runs as it comes (on the pieces' own memory), and the piece is recorded anew.
    for (int attempt = 0; ok && !s.pieces[k].e; ++attempt) {
      ok = attempt < 3 && record_begin();
      if (!ok) break;
      fresh();
      spoiled = false;
      memcpy(gr.base_counters, r.counters, sizeof(gr.base_counters));
      copies0 = r.main_copies;
      chains0 = trace_fused_chains();
      make_piece(p, piece, at, images[k], hosts);
      if (spoiled) continue;
      if (k + 1 == pieces) {
        enqueue_copy(n->result.aside, n->result.tensor, n->result.bytes, r.stream);
        enqueue_copy(n->result.tensor, n->result.made, n->result.bytes, r.stream);
      }
      ok = !spoiled && record_end(&s.pieces[k].e, false) && s.pieces[k].e;
    }
    if (!ok) break;
    for (int i = 0; i < CNT_COUNT; ++i) s.counters[i] += r.counters[i] - gr.base_counters[i];
    s.copies += r.main_copies - copies0;
    s.chains += trace_fused_chains() - chains0;
  }
  gr.making_pieces = false;
  s.counters[CNT_H2D_SKIPPED] = s.counters[CNT_POOL_HWM] = 0;
  cudaGetLastError();
  reg_drop_range((void *)mine, gr.piece_bytes);
  restore_registry(v.segments.back().after, v.pool_base, trace_pool_bytes());
  memcpy(r.counters, counters, sizeof(counters));
  r.main_copies = copies;
  if (!ok || epoch != gr.epoch) return;
  // of the pool's tensors the result alone is there afterwards
  for (const SavedRec &o : v.segments.back().after) {
    SavedRec rec = o;
    if (v.pool_base + o.offset != c.out - p.pool_base + v.pool_base && o.rec.fmt != FMT_PENDING && o.rec.fmt != FMT_ZERO) {
      rec.rec.fmt = FMT_ELIDED;
      rec.rec.home = rec.rec.dev_src = nullptr;
    }
    s.after.push_back(rec);
  }
  n->epoch = gr.epoch;
  n->used = ++gr.tick;
  GR_LOG("window cut up: %lld images\n", (long long)c.batch);
  add_variant(plan, std::move(n));
  plan.piece_failures = 0;
}

void launch_segment() {
  Runtime &r = rt();
  Variant &v = *gr.left[0];
  const Segment &s = v.segments[gr.seg];
  gr.left.resize(1);   // the others may differ from here on
  if (v.pieces) {
    for (int i = 0; i < MAX_PIECES && s.pieces[i].e; ++i) {
      if (i < gr.pieces_coming) OCC_CUDA(cudaStreamWaitEvent(r.stream, gr.piece_here[i], 0));
      OCC_CUDA(cudaGraphLaunch(s.pieces[i].e, r.stream));
    }
    gr.pieces_coming = 0;
  } else {
    wait_for_upload();
    if (s.exec.e) OCC_CUDA(cudaGraphLaunch(s.exec.e, r.stream));
  }
  for (int i = 0; i < CNT_COUNT; ++i) r.counters[i] += s.counters[i];
  r.main_copies += s.copies;
  for (int64_t i = 0; i < s.chains; ++i) trace_count_chain();
  if (gr.seg == 0) count(v.pieces ? CNT_IN_PIECES : CNT_REPLAYED);
  if (++gr.seg == v.segments.size()) {   // the window is done: later calls run one by one
    restore_registry(s.after, trace_pool_base(), trace_pool_bytes());
    trace_adopt_prefix(gr.prog, gr.prog->graph->end);
    v.used = ++gr.tick;
    gr.state = PLAIN;
    gr.left.clear();
    if (v.pieces) {
      gr.in_pieces = gr.prog;
      gr.pieces_of = &v;
    } else {
      build_pieces(*gr.prog, v);
    }
  }
}

// Graphs write into buffers of the runtime's that were free when they were captured.  The values of this
// inference's tensors that are in such buffers are compared (same_registry); those of tensors outside the pool
// move to their tensors' own memory.
void clear_homes(uintptr_t base, size_t bytes) {
  std::vector<uintptr_t> all;
  for (const auto &kv : rt().recs)
    if (kv.second.home && (kv.first < base || kv.first >= base + bytes)) all.push_back(kv.first);
  for (uintptr_t p : all) ensure_f32((const void *)p);
}

void start_window() {
  gr.prog = trace_candidate();
  GraphPlan &plan = *gr.prog->graph;
  const uintptr_t base = trace_pool_base();
  clear_homes(base, trace_pool_bytes());
  auto select = [&](bool pieces) {
    gr.left.clear();
    for (auto &v : plan.variants)
      if (v->pool_base == base && v->flags == mode_flags() && v->epoch == gr.epoch && v->pieces == pieces &&
          same_registry(v->before, base, trace_pool_bytes()))
        gr.left.push_back(v.get());
  };
  select(gr.pieces_coming > 0);
  if (gr.pieces_coming && gr.left.empty()) {
    wait_for_upload();
    select(false);
  }
  gr.next = plan.begin;
  gr.seg = gr.constant = 0;
  if (!gr.left.empty()) {
    gr.hosts.assign(plan.end - plan.begin, nullptr);
    gr.state = REPLAYING;
  } else if (plan.ready && plan.failures < MAX_FAILURES) {
    gr.building.reset(new Variant);
    gr.building->pool_base = base;
    gr.building->flags = mode_flags();
    gr.building->epoch = gr.epoch;
    save_registry(gr.building->before, base, trace_pool_bytes());
    if (!begin_segment()) {
      gr.building.reset();
      gr.state = PLAIN;
    }
  } else {
    gr.state = PLAIN;
  }
}

}  // namespace

void enqueue_kernel(const void *kernel, const cudaLaunchConfig_t &cfg, void **args) {
  if (recording && cfg.stream == rt().stream) {
    if (record_kernel(kernel, cfg, args)) return;
    graph_stop_capture();
  }
  cudaLaunchKernelExC(&cfg, kernel, args);
}

void enqueue_copy(void *dst, const void *src, size_t bytes, cudaStream_t s) {
  if (recording && s == rt().stream) {
    if (record_copy(dst, src, bytes)) return;
    graph_stop_capture();
  }
  OCC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s));
}

void enqueue_zero(void *dst, size_t bytes, cudaStream_t s) {
  if (recording && s == rt().stream) {
    if (record_copy(dst, nullptr, bytes)) return;
    graph_stop_capture();
  }
  OCC_CUDA(cudaMemsetAsync(dst, 0, bytes, s));
}

bool graph_upload_in_pieces(void *dst, const void *src, size_t bytes, cudaStream_t copy_stream) {
  if (gr.state != IDLE || !allowed()) return false;
  TraceProgram *p = trace_candidate();
  if (!p || !p->graph || trace_index() != p->graph->begin) return false;
  const uintptr_t base = trace_pool_base();
  bool there = false;
  for (auto &v : p->graph->variants)
    there = there || (v->pieces && v->pool_base == base && v->flags == mode_flags() && v->epoch == gr.epoch);
  Cut c;
  int64_t images[MAX_PIECES];
  if (!there || !find_input(*p, c) || (size_t)c.x_bytes != bytes || c.x - p->pool_base + base != (uintptr_t)dst) return false;
  const int pieces = piece_images(c.batch, images);
  if (!pieces) return false;
  for (cudaEvent_t &e : gr.piece_here)
    if (!e) OCC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  size_t at = 0;
  for (int k = 0; k < pieces; ++k) {
    const size_t n = bytes / (size_t)c.batch * (size_t)images[k];
    OCC_CUDA(cudaMemcpyAsync((char *)dst + at, (const char *)src + at, n, cudaMemcpyHostToDevice, copy_stream));
    OCC_CUDA(cudaEventRecord(gr.piece_here[k], copy_stream));
    at += n;
  }
  gr.pieces_coming = pieces;
  return true;
}

void graph_uncovered() { wait_for_upload(); }

void graph_left_recording() {
  TraceProgram *p = gr.in_pieces;
  if (!p || !trace_pool_base()) return;
  gr.in_pieces = nullptr;
  const Variant &v = *gr.pieces_of;
  const uintptr_t base = trace_pool_base();
  const std::vector<const void *> hosts = gr.hosts;
  enqueue_copy(v.result.tensor, v.result.aside, v.result.bytes, rt().stream);
  restore_registry(v.before, base, trace_pool_bytes());
  gr.again = true;
  for (size_t i = p->graph->begin; i < p->graph->end; ++i) {
    trace_force(p->roles[i]);
    run_again(p->entries[i],
              [&](void *q) {
                const uintptr_t a = (uintptr_t)q;
                return (void *)(a >= p->pool_base && a < p->pool_base + p->pool_bytes ? a - p->pool_base + base : a);
              },
              hosts[i - p->graph->begin]);
  }
  trace_force_end();
  flush_held_back();
  gr.again = false;
}

void graph_free_memory() {
  if (!gr.piece_memory || gr.making_pieces) return;
  graph_forget_all();
  OCC_CUDA(cudaStreamSynchronize(rt().stream));
  OCC_CUDA(cudaFree(gr.piece_memory));
  gr.piece_memory = nullptr;
  gr.piece_bytes = 0;
}

bool graph_covers(const Entry &e) {
  if (gr.state != REPLAYING) return false;
  TraceProgram *p = gr.prog;
  bool same = p->sigs[gr.next] == e.sig;
  if (same && e.sym == S_H2D) {
    const uint64_t hash = (uint64_t)e.args.v[1];
    size_t keep = 0;
    Variant *const leader = gr.left[0];
    for (Variant *v : gr.left) {
      const Constant &c = v->constants[gr.constant];
      if (c.src == e.host && c.hash == hash) gr.left[keep++] = v;
    }
    if (keep == 0) {
      gr.left.assign(1, leader);   // whose graphs have been launched so far
      same = false;
    } else {
      gr.left.resize(keep);
      ++gr.constant;
      gr.hosts[gr.next - p->graph->begin] = e.host;
      count(CNT_H2D_SKIPPED, e.args.v[0]);
    }
  }
  if (!same) {
    take_back();
    return false;
  }
  ++gr.next;
  while (gr.state == REPLAYING && gr.next >= gr.left[0]->segments[gr.seg].end) launch_segment();
  return true;
}

void graph_after_call() {
  if (gr.again || gr.state == PLAIN || gr.state == REPLAYING) return;
  if (gr.state == CAPTURING) {
    TraceProgram *p = trace_candidate();
    if (p != gr.prog || gr.epoch != gr.building->epoch) {
      graph_stop_capture();
      return;
    }
    const size_t n = trace_index();
    GraphPlan &plan = *p->graph;
    const bool cut = gr.building->segments.empty() && !anything_held_back() && computes(p->entries[n - 1].sym) &&
                     rt().counters[CNT_LAUNCHES] - gr.base_counters[CNT_LAUNCHES] >= FIRST_GRAPH_LAUNCHES;
    if (n == plan.end || cut) close_segment(plan);
    return;
  }
  // IDLE: the window may begin with the next call
  TraceProgram *p = trace_candidate();
  if (p && p->graph && trace_index() == p->graph->begin) {
    if (allowed()) start_window();
    else gr.state = PLAIN;
  }
}

static void break_capture() {
  if (recording && gr.state != CAPTURING) {   // of a piece: none of it is wanted
    cudaGraphDestroy(recording->graph);
    delete recording;
    recording = nullptr;
    spoiled = true;
    return;
  }
  if (gr.state != CAPTURING) return;
  GR_LOG("capture broken off at call %zu\n", trace_index());
  Exec launched;
  end_segment(&launched.e);
  gr.building.reset();
  if (gr.prog && gr.prog->graph) gr.prog->graph->failures++;
}

void graph_stop_capture() {
  gr.disturbed = true;
  break_capture();
}

void graph_before_upload() { break_capture(); }

void graph_settle() {
  if (gr.state == REPLAYING) take_back();
  else break_capture();
  wait_for_upload();   // it is among the calls made so far
}

void graph_forget_all() {
  gr.epoch++;
  gr.disturbed = true;
  break_capture();
}

void graph_inference_begin() {
  graph_settle();
  wait_for_upload();
  empty_trash(gr.trash.size() > 64);
  gr.state = IDLE;
  gr.prog = gr.in_pieces = nullptr;
  gr.disturbed = false;
  gr.epoch_at_begin = gr.epoch;
}

void graph_inference_end() {
  graph_settle();
  GR_LOG("end: cand %d own %d index %zu epoch %d disturbed %d\n", trace_candidate() != nullptr, (int)trace_has_own_entries(),
         trace_index(), (int)(gr.epoch - gr.epoch_at_begin), (int)gr.disturbed);
  // a complete inference made call by call, quietly, of a known program: its window may be captured
  TraceProgram *p = trace_candidate();
  if (trace_active() && p && trace_has_own_entries() && p->sigs.size() == trace_index() &&
      gr.epoch == gr.epoch_at_begin && !gr.disturbed)
    look_for_window(trace_entries(), *p);
  gr.in_pieces = nullptr;
  gr.state = PLAIN;
}

}  // namespace occ
