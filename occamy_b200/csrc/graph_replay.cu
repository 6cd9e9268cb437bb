// Capture, matching and launch of recorded inferences (see graph_replay.h).
#include "graph_replay.h"

#include <cstring>
#include <map>

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

struct Segment {
  cudaGraphExec_t exec = nullptr;   // null: the calls enqueue nothing
  size_t end = 0;                   // one past its last call
  std::vector<SavedRec> after;      // registry records of the pool when it has been enqueued
  int64_t counters[8] = {};         // what its calls count
  int64_t copies = 0, chains = 0;
};

struct Constant {
  size_t call;
  const void *src;
  uint64_t hash;
};

struct Variant {
  uintptr_t pool_base = 0;
  int flags = 0;
  uint64_t epoch = 0, used = 0;
  std::vector<SavedRec> before;   // the pool's records when the window began: the forms its inputs are in
  std::vector<Constant> constants;
  std::vector<Segment> segments;
};

}  // namespace

struct GraphPlan {
  size_t begin = 0, end = 0;   // the window: calls [begin, end)
  bool ready = false;          // an inference ran with nothing to upload or allocate inside it
  int failures = 0;
  std::vector<std::unique_ptr<Variant>> variants;
  ~GraphPlan();
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
  int64_t base_counters[8] = {};
  int64_t base_copies = 0, base_chains = 0;
  std::vector<cudaGraphExec_t> trash;   // launched once, destroyed when the stream is idle
};
Replay &gr = *new Replay;   // never destroyed, like the programs it refers to

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

bool same_registry(const std::vector<SavedRec> &a, uintptr_t base, size_t bytes) {
  auto &recs = rt().recs;
  auto it = recs.lower_bound(base);
  for (const SavedRec &s : a) {
    if (it == recs.end() || it->first != base + s.offset || it->second.fmt != s.rec.fmt || it->second.home != s.rec.home)
      return false;
    ++it;
  }
  return it == recs.end() || it->first >= base + bytes;
}

// ---- capture --------------------------------------------------------------------
bool begin_segment() {
  Runtime &r = rt();
  memcpy(gr.base_counters, r.counters, sizeof(gr.base_counters));
  gr.base_copies = r.main_copies;
  gr.base_chains = trace_fused_chains();
  // relaxed: other threads and libraries of the process go on allocating meanwhile
  const cudaError_t e = cudaStreamBeginCapture(r.stream, cudaStreamCaptureModeRelaxed);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  gr.state = CAPTURING;
  return true;
}

// Ends the capture and launches what it holds.  The executable graph, or null when it is empty.
bool end_segment(cudaGraphExec_t *exec) {
  Runtime &r = rt();
  *exec = nullptr;
  gr.state = PLAIN;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(r.stream, &g);
  size_t nodes = 0;
  if (e == cudaSuccess && g) e = cudaGraphGetNodes(g, nullptr, &nodes);
  if (e == cudaSuccess && nodes) e = cudaGraphInstantiate(exec, g, 0);
  if (e == cudaSuccess && *exec) e = cudaGraphLaunch(*exec, r.stream);
  if (g) cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    set_error((int)e, "capture of a recorded inference");
    return false;
  }
  return true;
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
  for (int i = 0; i < 8; ++i) s.counters[i] = r.counters[i] - gr.base_counters[i];
  s.counters[CNT_H2D_SKIPPED] = s.counters[CNT_POOL_HWM] = 0;   // counted as the calls are checked
  s.copies = r.main_copies - gr.base_copies;
  s.chains = trace_fused_chains() - gr.base_chains;
  save_registry(s.after, trace_pool_base(), trace_pool_bytes());
  if (!end_segment(&s.exec)) {
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
    run_again(p->entries[i], (intptr_t)(base - p->pool_base), p->pool_base, p->pool_bytes,
              gr.hosts[i - p->graph->begin]);
  gr.again = false;
}

void launch_segment() {
  Runtime &r = rt();
  Variant &v = *gr.left[0];
  const Segment &s = v.segments[gr.seg];
  gr.left.resize(1);   // the others may differ from here on
  if (s.exec) OCC_CUDA(cudaGraphLaunch(s.exec, r.stream));
  for (int i = 0; i < 8; ++i) r.counters[i] += s.counters[i];
  r.main_copies += s.copies;
  for (int64_t i = 0; i < s.chains; ++i) trace_count_chain();
  if (++gr.seg == v.segments.size()) {   // the window is done: later calls run one by one
    restore_registry(s.after, trace_pool_base(), trace_pool_bytes());
    trace_adopt_prefix(gr.prog, gr.prog->graph->end);
    v.used = ++gr.tick;
    gr.state = PLAIN;
    gr.left.clear();
  }
}

void start_window() {
  gr.prog = trace_candidate();
  GraphPlan &plan = *gr.prog->graph;
  const uintptr_t base = trace_pool_base();
  gr.left.clear();
  for (auto &v : plan.variants)
    if (v->pool_base == base && v->flags == mode_flags() && v->epoch == gr.epoch &&
        same_registry(v->before, base, trace_pool_bytes()))
      gr.left.push_back(v.get());
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

GraphPlan::~GraphPlan() {
  for (auto &v : variants)
    for (Segment &s : v->segments)
      if (s.exec) gr.trash.push_back(s.exec);
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
  if (gr.state != CAPTURING) return;
  GR_LOG("capture broken off at call %zu\n", trace_index());
  cudaGraphExec_t e = nullptr;
  end_segment(&e);
  if (e) gr.trash.push_back(e);
  for (Segment &s : gr.building->segments)
    if (s.exec) gr.trash.push_back(s.exec);
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
}

void graph_forget_all() {
  gr.epoch++;
  gr.disturbed = true;
  break_capture();
}

void graph_inference_begin() {
  graph_settle();
  empty_trash(gr.trash.size() > 64);
  gr.state = IDLE;
  gr.prog = nullptr;
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
  gr.state = PLAIN;
}

}  // namespace occ
