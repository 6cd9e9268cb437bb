// The C-ABI entry points on the CNN hot path (declared in include/occamy_dnn_api.h) and
// the dispatch between the fp32 NCHW kernels and the bf16 NHWC / tensor-core kernels.
#include <cstring>
#include <initializer_list>
#include <vector>

#include "graph_replay.h"
#include "kernels.h"
#include "runtime.h"
#include "trace.h"

#define OCCAMY_NO_VENDOR_TYPES
typedef cudaError_t occamy_cuda_error_t;
struct cudnnContext;
typedef struct cudnnContext *cudnnHandle_t;
#include "../../include/occamy_dnn_api.h"

using namespace occ;

namespace {

struct PoolRec {
  void *base;
  size_t bytes;
};
std::vector<PoolRec> g_pools;
// Pool blocks of finished inferences, kept so that the next wrapDNNMemPoolInit of the same
// size costs no cudaMalloc / cudaFree (a compiled model creates and frees its pool on every
// call).  Up to OCCAMY_POOL_BLOCKS (default 2, 0 = off) blocks of one size are kept and
// handed out in turn: consecutive inferences then live in different blocks, and the input
// upload of the next one can run on the copy stream while the kernels of the current one
// are still executing.
struct CachedPool {
  void *base;
  size_t bytes;
  cudaEvent_t done;   // recorded on the launch stream when the block's last user finished
};
std::vector<CachedPool> g_pool_cache;   // oldest first
cudaEvent_t g_block_ready = nullptr;    // `done` of the block the current inference lives in
void *g_cur_pool = nullptr;
size_t g_cur_pool_bytes = 0;
cudaStream_t g_copy_stream = nullptr;
int64_t g_launches_at_pool_init = 0;   // kernel + copy count when the current pool was set up

int pool_cache_blocks() {
  static int v = -1;
  if (v < 0) {
    const char *e = getenv("OCCAMY_POOL_BLOCKS");
    if (!e) e = getenv("OCCAMY_POOL_CACHE");
    v = e ? atoi(e) : 2;
    if (v < 0) v = 0;
    if (v > 4) v = 4;
  }
  return v;
}

void free_cached_pool(CachedPool &c) {
  OCC_CUDA(cudaEventSynchronize(c.done));
  OCC_CUDA(cudaFree(c.base));
  OCC_CUDA(cudaEventDestroy(c.done));
}

void die(const char *what, cudaError_t e, size_t size) {
  // Same convention as the reference's memory wrappers (cuda/wrapDNNMalloc.cpp:11-16).
  printf("[%s] GPU error: (size: %zu) %s\n", what, size, cudaGetErrorString(e));
  exit(-1);
}

enum PackLayout { PACK_KRSC = 1, PACK_DW = 2, PACK_FOLD = 3, PACK_RAW = 4, PACK_STEM = 5, PACK_PARTS = 6, PACK_BIAS3 = 7, PACK_IR_HALF = 8 };
// fp32 mode: dense convolutions and GEMMs on the tensor cores with split operands (see
// kernels_parts.cu); off with OCCAMY_FP32_TC=0 or occamy_set_fp32_tensor_cores(0), which
// leaves the CUDA-core kernels.
int g_fp32_tc = -1;
}  // namespace
bool occ::fp32_on_tensor_cores() {
  if (g_fp32_tc < 0) {
    const char *e = getenv("OCCAMY_FP32_TC");
    g_fp32_tc = (e && !strcmp(e, "0")) ? 0 : 1;
  }
  return g_fp32_tc == 1;
}
namespace {

// Device pointer of the packed form of the filter at `w`; resident across calls when the
// filter was uploaded from host memory (a compiled model's constant), otherwise packed
// into scratch.  `packed_bytes` is the size of the packed form.
// Set by packed_weights: the returned copy was already on the device before this call (no
// kernel or copy was enqueued to produce it).
bool g_pack_was_resident = false;

void *packed_weights(const float *w, int layout, size_t packed_bytes, int K, int C, int R, int S,
                     int Sp, int Cp) {
  Runtime &r = rt();
  g_pack_was_resident = false;
  uintptr_t base;
  TensorRec *rec = reg_find(w, &base);
  const bool cacheable = r.cache_weights && rec && base == (uintptr_t)w && rec->host_src;
  // fp32 layouts are shared by the two 16-bit modes, 16-bit ones are packed per element type
  const bool f16 = mode_f16() && layout != PACK_DW && layout != PACK_RAW && layout != PACK_PARTS;
  WeightKey key{nullptr, 0, layout * 4096 + Sp * 64 + Cp + (f16 ? (1 << 20) : 0)};
  if (cacheable) {
    key.src = rec->host_src;
    key.bytes = rec->host_bytes;
    auto it = r.wcache.find(key);
    if (it != r.wcache.end() && it->second.hash == rec->host_hash && it->second.bytes == packed_bytes) {
      g_pack_was_resident = true;
      r.resident[key.src] = std::make_pair(key.bytes, it->second.hash);   // (another constant may have been there since)
      return it->second.dev;
    }
  }
  void *dst = nullptr;
  if (cacheable) {
    graph_stop_capture();   // packed once, not in every inference
    if (rec->fmt == FMT_PENDING) {
      // Not on the device: it goes through a buffer of the runtime's.  (Its own place may still hold what a
      // held-back kernel has to read.)
      void *tmp = scratch_get(8, rec->host_bytes);
      if (!tmp) return nullptr;
      OCC_CUDA(cudaMemcpyAsync(tmp, rec->host_src, rec->host_bytes, cudaMemcpyHostToDevice, r.stream));
      r.main_copies++;
      count(CNT_H2D_BYTES, (int64_t)rec->host_bytes);
      w = (const float *)tmp;
    } else {
      ensure_f32(w);
    }
    PackedWeight &pw = r.wcache[key];
    if (pw.dev) graph_forget_all();   // graphs refer to the old contents
    if (pw.dev && pw.bytes != packed_bytes) {
      OCC_CUDA(cudaStreamSynchronize(r.stream));
      OCC_CUDA(cudaFree(pw.dev));
      pw.dev = nullptr;
    }
    if (!pw.dev) OCC_CUDA(device_malloc(&pw.dev, packed_bytes));
    pw.bytes = packed_bytes;
    pw.hash = rec->host_hash;
    pw.layout = layout;
    dst = pw.dev;
    r.resident[rec->host_src] = std::make_pair(rec->host_bytes, rec->host_hash);
  } else {
    ensure_f32(w);
    dst = scratch_get(layout == PACK_STEM ? 5 : 1, packed_bytes);
  }
  if (!dst) return nullptr;
  if (layout == PACK_KRSC) launch_pack_krsc_bf16(w, (bf16 *)dst, K, C, R, S, Cp, f16, r.stream);
  else if (layout == PACK_DW) launch_pack_dw_f32(w, (float *)dst, C, R, S, r.stream);
  else if (layout == PACK_RAW)
    enqueue_copy(dst, w, packed_bytes, r.stream);
  else if (layout == PACK_STEM) launch_pack_stem_bf16(w, (bf16 *)dst, C, R, S, Cp, Sp * Cp, r.stream);
  else if (layout == PACK_BIAS3) launch_pack_bias3(w, (bf16 *)dst, K, f16, r.stream);
  else if (layout == PACK_IR_HALF) launch_pack_ir_half(w, dst, K, R * S, r.stream);
  else if (layout == PACK_PARTS) launch_pack_split3(w, (bf16 *)dst, K, C, R, S, Sp, Cp, r.stream);
  else launch_pack_fold_bf16(w, (bf16 *)dst, K, C, R, S, Sp, Cp, f16, r.stream);
  return dst;
}

// Whether the packed form of `p` stays on the device.  One that does not is packed into scratch, where the next
// one replaces it: its convolution has to be launched before another is prepared.
bool stays_packed(const float *p) {
  uintptr_t base;
  const TensorRec *rec = reg_find(p, &base);
  return rt().cache_weights && rec && base == (uintptr_t)p && rec->host_src;
}

// A constant in the form the inverted-residual kernel takes it (the first convolution's bias as parts; the
// depthwise filter or bias as fp16); null unless it stays on the device.
const void *packed_for_block(const float *c, int layout, size_t bytes, int E, int R) {
  if (!stays_packed(c)) return nullptr;
  return packed_weights(c, layout, bytes, E, 0, R, R, 0, 0);
}

// fp32 constants used as they are (biases mostly): the resident copy when there is one, else the
// tensor itself.
const float *resident_f32(const float *p, size_t bytes) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  if (rt().cache_weights && rec && base == (uintptr_t)p && rec->host_src && rec->host_bytes == bytes) {
    const float *d = (const float *)packed_weights(p, PACK_RAW, bytes, 0, 0, 0, 0, 0, 0);
    if (d) return d;
  }
  g_pack_was_resident = false;
  ensure_f32(p);
  return p;
}

// The second operand of an element-wise call or of a product, the filter of a convolution on the CUDA cores.
// It may be an input of the model as well as a constant, and of a large one the fingerprint is a sample: those are
// read from the tensor itself, uploaded in full every time.
const float *operand_f32(const float *p, size_t bytes) {
  if (bytes <= HASH_WHOLE) return resident_f32(p, bytes);
  ensure_f32(p);
  return p;
}

// ---- a convolution resolved down to launch arguments ------------------------------
// `prepare_*` does everything that depends on the inputs' current state (layout
// conversion into scratch, packed-weight lookup, bias lookup); what is left is a launch
// that only needs to be told where to write, which residual to add and how to clamp.
struct ConvJob {
  bool active = false;
  bool depthwise = false;
  ConvGeom g;
  TcConvArgs a = {};          // dense: tensor-core arguments (x, w, bias resolved)
  const bf16 *dw_x = nullptr; // depthwise
  const float *dw_w = nullptr;
  const float *bias = nullptr;
  float *out = nullptr;       // tensor the result goes to
  bool bias_set = false, res_set = false, act_set = false;
  int absorbed = 0;           // later calls folded into this one so far
  // device ranges still to be read: [0] input, [1] residual operand, [2] a bias that is read
  // from the caller's tensor (no resident copy exists)
  // ([3], [4]: input and bias of a second summand)
  uintptr_t dep_lo[5] = {}, dep_hi[5] = {};
  // a matrix product: `g` says N x K results (P = Q = 1), `a` how they are computed
  bool product = false;
  bool out16 = false;             // ... whose reader is another product: 16-bit result
  // fp32 mode (a.split): the result goes out in three planes (FMT_PARTS), else as plain fp32
  bool out_parts = false;
  // one of the convolutions of an inverted residual: its result only goes to the next one / its input
  // only comes from the one before (and is not there yet)
  bool linked = false, joined = false;
  // held back until a sum takes its result along (RF_SUM) / the other summand, which g_front[0] still is
  bool summand = false, after_summand = false;
  // its result is read by the convolution behind it (RF_LEAD) / the one in front, g_front[0], writes its input
  bool leads = false, follows = false;
  // (the constants of one once more, packed_for_block(): a first bias, a depthwise filter and bias)
  const void *block_w = nullptr, *block_b = nullptr;
  // folded (few-channel) form: what the fused convolution + pool kernel needs besides `a`
  const bf16 *w_stem = nullptr;   // filter in that kernel's layout, packed while the filter is live
};

ConvJob g_pending;  // convolution held back while later calls are folded into it
ConvJob g_front[2]; // ... and the ones before it that it has joined, not launched yet either
int g_fronts = 0;
const ConvJob *g_launching = nullptr;   // job whose output buffer is being looked for

bool job_reads(const ConvJob &j, const void *home) {
  return j.a.x == home || j.a.y == home || j.a.x2 == home || j.a.residual == home || j.dw_x == home;
}
bool home_held_hook(const void *home) {
  for (int i = 0; i < g_fronts; ++i)
    if (job_reads(g_front[i], home)) return true;
  return ((g_pending.active || g_fronts) && job_reads(g_pending, home)) ||
         (g_launching && job_reads(*g_launching, home));
}

// A bias without a resident copy is read from the caller's tensor when the (possibly held-back)
// kernel finally runs: until then that tensor must neither be freed nor overwritten.
void job_track_bias(ConvJob &job, const float *used, const float *callers, int channels) {
  job.dep_lo[2] = job.dep_hi[2] = 0;
  if (used && used == callers) {
    job.dep_lo[2] = (uintptr_t)callers;
    job.dep_hi[2] = (uintptr_t)callers + (size_t)channels * 4;
  }
}

// The folded form of a few-channel convolution: channels padded so that one output column's step along
// the row is a multiple of 16 bytes, width taps padded to whole steps, pixels per padded row.
void stem_geometry(const ConvGeom &g, int &Cp, int &Sp, int &Wp) {
  Cp = g.C <= 4 ? (g.stride_w % 2 == 0 ? 4 : 8) : (g.C <= 8 ? 8 : 16);
  const int unit = 16 / Cp;
  Sp = (g.S + unit - 1) / unit * unit;
  Wp = g.pad_w + g.W;
  if (Wp < (g.Q - 1) * g.stride_w + Sp) Wp = (g.Q - 1) * g.stride_w + Sp;
  Wp = (Wp + 7) / 8 * 8;
}

// TcConvArgs::form_n of a convolution on n images, a product of n rows.
int form_n(int64_t n) { return form_images(n) == n ? 0 : (int)form_images(n); }

// A dense convolution of the 16-bit path as the kernels are told of it, but for where its operands are;
// false when they do not take it.  Cp, Sp, Wp: how the input is stored (stem_geometry(), when it is folded).
bool dense_args(const ConvGeom &g, TcConvArgs &a, int &Cp, int &Sp, int &Wp) {
  memset(&a, 0, sizeof(a));
  if (g.groups != 1 || g.K % 8 != 0) return false;
  if (g.act != ACT_IDENTITY && g.act != ACT_RELU && g.act != ACT_CLIP) return false;
  a.N = g.N; a.K = g.K; a.P = g.P; a.Q = g.Q;
  a.form_n = form_n(g.N);
  a.act = g.act; a.lo = g.lo; a.hi = g.hi;
  a.f16 = mode_f16() ? 1 : 0;
  Sp = Cp = Wp = 0;
  if (g.C < 16) {
    stem_geometry(g, Cp, Sp, Wp);
    a.H = g.H; a.W = g.Q; a.Cf = Sp * Cp;
    a.R = g.R; a.S = 1;
    a.pad_h = g.pad_h; a.pad_w = 0; a.stride_h = g.stride_h; a.stride_w = 1;
    a.w_step = g.stride_w * Cp;
    a.row_elems = Wp * Cp;
  } else {
    if (g.C % 8 != 0) return false;
    // Pixels are padded to a multiple of 32 bytes with zero channels: rows at a 48-byte pitch
    // (24 channels) load at little more than half the speed of rows at 64 (measured:
    // 24->144 at 56x56, 0.044 ms padded, 0.072 ms not).
    Cp = (g.C + 15) / 16 * 16;
    a.H = g.H; a.W = g.W; a.Cf = Cp;
    a.R = g.R; a.S = g.S;
    a.pad_h = g.pad_h; a.pad_w = g.pad_w; a.stride_h = g.stride_h; a.stride_w = g.stride_w;
  }
  a.x = (const bf16 *)16;  // placeholders so the support check sees aligned pointers
  a.w = (const bf16 *)16;
  a.y = (bf16 *)16;
  return tc_conv_supported(a);
}

// `job.linked` (the first convolution of an inverted residual): x is taken as it is, without the padding of
// its channels; `job.joined`: x is not there yet.
bool prepare_dense(const float *x, const float *w, const float *bias, const ConvGeom &g,
                   ConvJob &job) {
  Runtime &r = rt();
  TcConvArgs &a = job.a;
  int Sp, Cp, Wp;
  if (!dense_args(g, a, Cp, Sp, Wp)) return false;
  const bool folded = g.C < 16;

  job.dep_lo[0] = job.dep_hi[0] = 0;
  if (folded) {
    uintptr_t base = 0;
    const TensorRec *rec = reg_find(x, &base);
    if (rec && base == (uintptr_t)x && rec->fmt == FMT_STEM_ROWS && rec->n == g.N && rec->c == g.C && rec->h == g.H &&
        rec->w == g.W && rec->stem_wp == Wp && rec->stem_cp == Cp && rec->stem_pad == g.pad_w &&
        rec->stem_f16 == (int)mode_f16()) {
      a.x = (const bf16 *)rec->home;   // brought in in this form
    } else {
      ensure_f32(x);
      bf16 *xf = (bf16 *)scratch_get(0, (size_t)g.N * g.H * Wp * Cp * 2);
      if (!xf) return false;
      launch_pad_input_bf16(x, xf, g.N, g.C, g.H, g.W, Wp, Cp, g.pad_w, mode_f16(), r.stream);
      a.x = xf;
    }
    a.w = (const bf16 *)packed_weights(w, PACK_FOLD, (size_t)g.R * g.K * a.Cf * 2, g.K, g.C, g.R,
                                       g.S, Sp, Cp);
  } else {
    const bf16 *xb = nullptr;
    const bool as_is = job.linked || job.joined;
    if (job.joined) {
      // (resolved when it is launched)
    } else if (is_act16(x, g.N, g.C, g.H, g.W)) {
      xb = act16_ptr(x);
      if ((Cp == g.C || as_is) && (const void *)xb == x) {
        job.dep_lo[0] = (uintptr_t)x;
        job.dep_hi[0] = (uintptr_t)x + (size_t)g.N * g.C * g.H * g.W * 2;
      }
    } else {
      ensure_f32(x);
      bf16 *xc = (bf16 *)scratch_get(0, (size_t)g.N * g.C * g.H * g.W * 2);
      if (!xc) return false;
      launch_nchw_f32_to_nhwc_bf16(x, xc, g.N, g.C, g.H, g.W, mode_f16(), r.stream);
      xb = xc;
    }
    if (Cp != g.C && !as_is) {   // the kernel reads the padded copy, made now: no dependence on x later
      bf16 *xp = (bf16 *)scratch_get(6, (size_t)g.N * Cp * g.H * g.W * 2);
      if (!xp) return false;
      launch_pad_channels_bf16(xb, xp, (int64_t)g.N * g.H * g.W, g.C, Cp, r.stream);
      xb = xp;
    }
    a.x = xb;
    a.w = (const bf16 *)packed_weights(w, PACK_KRSC, (size_t)g.R * g.S * g.K * Cp * 2, g.K, g.C,
                                       g.R, g.S, 0, Cp);
  }
  if (!a.w) return false;
  bool ready = g_pack_was_resident;
  a.bias = bias ? resident_f32(bias, (size_t)g.K * 4) : nullptr;
  if (bias) ready = ready && g_pack_was_resident;
  job_track_bias(job, a.bias, bias, g.K);
  if (bias && job.linked && !job.joined) {
    job.block_b = packed_for_block(bias, PACK_BIAS3, (size_t)g.K * 32, g.K, 0);
    ready = ready && g_pack_was_resident;
  }
  // filter and bias were on the device before this call: the kernel may fetch them while the
  // kernel before it is still running
  a.consts_ready = ready ? 1 : 0;
  job.depthwise = false;
  job.g = g;
  job.bias_set = bias != nullptr;
  job.act_set = g.act != ACT_IDENTITY;
  job.res_set = false;
  job.w_stem = nullptr;
  return true;
}

// fp32 mode on the tensor cores: x and the filter are carried as three bf16 parts each and the six part
// products that matter are accumulated in fp32 (conv_tc_split.cu).  False when the shape is outside what
// the kernel takes (the CUDA-core kernel runs then).
bool parts_shape_ok(const ConvGeom &g) {
  // Tiny problems stay on the CUDA-core kernel: the passes around this one cost more than it saves.
  return fp32_on_tensor_cores() && g.groups == 1 && g.R * g.S <= 64 && g.stride_h <= 2 && g.stride_w <= 2 &&
         (g.act == ACT_IDENTITY || g.act == ACT_RELU || g.act == ACT_CLIP) &&
         (double)form_images(g.N) * g.P * g.Q * g.K * g.C * g.R * g.S >= 1e6;
}

bool prepare_parts(const float *x, const float *w, const float *bias, const ConvGeom &g, ConvJob &job) {
  Runtime &r = rt();
  if (!parts_shape_ok(g)) return false;
  TcConvArgs &a = job.a;
  memset(&a, 0, sizeof(a));
  a.N = g.N; a.H = g.H; a.K = g.K; a.P = g.P; a.Q = g.Q; a.R = g.R;
  a.form_n = form_n(g.N);
  a.pad_h = g.pad_h; a.stride_h = g.stride_h;
  a.act = g.act; a.lo = g.lo; a.hi = g.hi;
  a.split = 1;
  a.out_nchw = 1;
  a.ldo = g.K;
  const bool folded = g.C < 16 && g.R <= 16;
  int Sp = 0, Cp = (g.C + 15) / 16 * 16, Wp = 0;
  if (folded) {
    stem_geometry(g, Cp, Sp, Wp);
    a.W = g.Q; a.Cf = Sp * Cp; a.S = 1;
    a.stride_w = 1;
    a.w_step = g.stride_w * Cp;
    a.row_elems = Wp * Cp;
  } else {
    a.W = g.W; a.Cf = Cp; a.S = g.S;
    a.pad_w = g.pad_w; a.stride_w = g.stride_w;
  }
  a.x = a.w = (const bf16 *)16;
  a.out_f32 = job.out;
  if (!tc_conv_supported(a)) return false;
  if (Cp == g.C && is_parts(x, g.N, g.C, g.H, g.W)) {
    a.x = act16_ptr(x);
  } else {
    ensure_f32(x);
    bf16 *xs = (bf16 *)scratch_get(0, (size_t)6 * g.N * g.H * (folded ? a.row_elems : g.W * Cp));
    if (!xs) return false;
    if (folded) launch_split3_pad(x, xs, g.N, g.C, g.H, g.W, Wp, Cp, g.pad_w, r.stream);
    else launch_split3_nchw(x, xs, g.N, g.C, Cp, g.H, g.W, r.stream);
    a.x = xs;
  }
  a.w = (const bf16 *)packed_weights(w, PACK_PARTS, (size_t)6 * a.R * a.S * g.K * a.Cf, g.K, g.C, g.R, g.S, Sp, Cp);
  if (!a.w) return false;
  bool ready = g_pack_was_resident;
  a.bias = bias ? resident_f32(bias, (size_t)g.K * 4) : nullptr;
  if (bias) ready = ready && g_pack_was_resident;
  a.consts_ready = ready ? 1 : 0;
  job_track_bias(job, a.bias, bias, g.K);
  job.g = g;
  job.bias_set = bias != nullptr;
  job.act_set = g.act != ACT_IDENTITY;
  return true;
}

bool prepare_depthwise(const float *x, const float *w, const float *bias, const ConvGeom &g,
                       ConvJob &job) {
  Runtime &r = rt();
  if (g.C % 8 != 0) return false;
  job.dep_lo[0] = job.dep_hi[0] = 0;
  if (job.joined) {
    job.dw_x = nullptr;
  } else if (is_act16(x, g.N, g.C, g.H, g.W)) {
    job.dw_x = act16_ptr(x);
    if ((const void *)job.dw_x == x) {
      job.dep_lo[0] = (uintptr_t)x;
      job.dep_hi[0] = (uintptr_t)x + (size_t)g.N * g.C * g.H * g.W * 2;
    }
  } else {
    ensure_f32(x);
    bf16 *xc = (bf16 *)scratch_get(0, (size_t)g.N * g.C * g.H * g.W * 2);
    if (!xc) return false;
    launch_nchw_f32_to_nhwc_bf16(x, xc, g.N, g.C, g.H, g.W, mode_f16(), r.stream);
    job.dw_x = xc;
  }
  job.dw_w = (const float *)packed_weights(w, PACK_DW, (size_t)g.R * g.S * g.C * 4, g.K, g.C, g.R,
                                          g.S, 0, 0);
  if (!job.dw_w) return false;
  bool ready = g_pack_was_resident;
  job.bias = bias ? resident_f32(bias, (size_t)g.C * 4) : nullptr;
  if (bias) ready = ready && g_pack_was_resident;
  if (job.linked && mode_f16()) {
    job.block_w = packed_for_block(w, PACK_IR_HALF, (size_t)g.C * 18, g.C, 3);
    ready = ready && g_pack_was_resident;
    if (bias) {
      job.block_b = packed_for_block(bias, PACK_IR_HALF, (size_t)g.C * 2, g.C, 1);
      ready = ready && g_pack_was_resident;
    }
  }
  job.a.consts_ready = ready ? 1 : 0;
  job_track_bias(job, job.bias, bias, g.C);
  job.depthwise = true;
  job.g = g;
  job.bias_set = bias != nullptr;
  job.act_set = g.act != ACT_IDENTITY;
  job.res_set = false;
  return true;
}

bool ranges_overlap(uintptr_t alo, uintptr_t ahi, uintptr_t blo, uintptr_t bhi) {
  return ahi > alo && bhi > blo && alo < bhi && blo < ahi;
}

// `apart`: the result goes to a buffer of its own, which is returned.
const bf16 *launch_job(ConvJob &job, bool apart = false) {
  Runtime &r = rt();
  const ConvGeom &g = job.g;
  // A convolution that was held back may find its output placed over memory it still has to read
  // (the planner reuses a tensor's bytes as soon as the recorded program no longer needs them).  The
  // result then goes to a buffer of its own, which the tensor's record points to; a residual operand
  // that the output covers exactly may stay (each tile reads its residual before it is stored).
  // (Copying the input out of the way instead cost 1.5 to 40 us per such layer and broke the chain of
  // overlapping launches: 17 copies in an unfused ResNet-50, 10 in MobileNetV2.)
  const uintptr_t olo = (uintptr_t)job.out;
  const size_t obytes = (size_t)g.N * g.K * g.P * g.Q * 2;
  const uintptr_t ohi = olo + obytes;
  void *dst = job.out;
  job.a.act = g.act; job.a.lo = g.lo; job.a.hi = g.hi;
  if (job.a.split && job.out_parts) {
    g_launching = &job;
    void *planes = home_acquire(obytes * 3);
    g_launching = nullptr;
    if (!planes) return nullptr;
    job.a.y = (bf16 *)planes;
    job.a.out_f32 = nullptr;
    launch_tc_conv(job.a, r.stream);
    mark_parts(job.out, g.N, g.K, g.P, g.Q, planes);
    return nullptr;
  }
  if (job.a.split || (job.product && !job.out16)) {   // fp32 result, at its own address
    for (int k = 0; k < 3; k += 2) {
      if (!ranges_overlap(olo, ohi + obytes, job.dep_lo[k], job.dep_hi[k])) continue;
      const size_t bytes = job.dep_hi[k] - job.dep_lo[k];
      void *tmp = scratch_get(k ? 7 : 4, bytes);
      enqueue_copy(tmp, (const void *)job.dep_lo[k], bytes, r.stream);
      if (k) job.a.bias = (const float *)tmp;
      else job.a.x = (const bf16 *)tmp;
      count(CNT_LAUNCHES);
    }
    job.a.out_f32 = job.out;
    job.a.ldo = g.K;
    job.a.out_nchw = !job.product || job.a.R * job.a.S > 1;   // (a product's [N][K][1][1]: the same rows)
    launch_tc_conv(job.a, r.stream);
    mark_f32(job.out);
    return nullptr;
  }
  const bool in_place = olo == job.dep_lo[1] && ohi == job.dep_hi[1];
  if (apart || ranges_overlap(olo, ohi, job.dep_lo[0], job.dep_hi[0]) ||
      (ranges_overlap(olo, ohi, job.dep_lo[1], job.dep_hi[1]) && !in_place) ||
      ranges_overlap(olo, ohi, job.dep_lo[2], job.dep_hi[2]) || ranges_overlap(olo, ohi, job.dep_lo[3], job.dep_hi[3]) ||
      ranges_overlap(olo, ohi, job.dep_lo[4], job.dep_hi[4])) {
    g_launching = &job;
    dst = home_acquire(obytes);
    g_launching = nullptr;
    if (!dst) return nullptr;
  }
  if (job.depthwise) {
    launch_depthwise_bf16(job.dw_x, job.dw_w, job.bias, (bf16 *)dst, g, mode_f16(), job.a.consts_ready != 0, r.stream);
  } else {
    job.a.y = (bf16 *)dst;
    launch_tc_conv(job.a, r.stream);
  }
  if (!apart) {
    mark_act16(job.out, g.N, g.K, g.P, g.Q, dst == job.out ? nullptr : dst);
  } else {   // its tensor may be gone by now: whoever joined this convolution was its only reader
    uintptr_t base;
    const TensorRec *rec = reg_find(job.out, &base);
    if (rec && base == olo && rec->fmt == FMT_ELIDED) mark_act16(job.out, g.N, g.K, g.P, g.Q, dst);
  }
  return (const bf16 *)dst;
}

// The three convolutions of an inverted residual in one kernel; false when they have to run one by one.
bool launch_block(ConvJob &a, ConvJob &b, ConvJob &c) {
  Runtime &r = rt();
  if (a.depthwise || !b.depthwise || c.depthwise || c.linked || !a.block_b) return false;
  IrArgs ir;
  memset(&ir, 0, sizeof(ir));
  const ConvJob *job[3] = {&a, &b, &c};
  for (int i = 0; i < 3; ++i) {
    const ConvGeom &g = job[i]->g;
    ir.floor[i] = g.act == ACT_RELU ? 0.0f : -INFINITY;
    ir.lo[i] = g.act == ACT_CLIP ? g.lo : NAN;
    ir.hi[i] = g.act == ACT_CLIP ? g.hi : NAN;
    if (g.act != ACT_IDENTITY && g.act != ACT_RELU && g.act != ACT_CLIP) return false;
  }
  const ConvGeom &g = c.g;
  ir.x = a.a.x; ir.w1 = a.a.w; ir.b1 = (const bf16 *)a.block_b;
  ir.w2 = b.dw_w; ir.b2 = b.bias;
  if (mode_f16()) {   // the kernel sums in fp16, which is for those depthwise convolutions that do so by themselves
    ir.w2 = b.block_w; ir.b2 = b.block_b;
    if (!depthwise_sums_in_half(b.g) || !ir.w2 || (b.bias && !ir.b2)) return false;
  }
  ir.w3 = c.a.w; ir.b3 = c.a.bias;
  ir.residual = c.a.residual;
  ir.N = g.N; ir.H = a.g.H; ir.W = a.g.W; ir.C = a.g.C; ir.E = a.g.K; ir.K = g.K; ir.P = g.P; ir.Q = g.Q;
  ir.stride = b.g.stride_h;
  ir.form_n = (int)form_images(g.N);
  ir.f16 = mode_f16();
  ir.consts_ready = a.a.consts_ready && b.a.consts_ready && c.a.consts_ready;
  if (!ir_supported(ir.form_n, ir.C, ir.E, ir.K, ir.H, ir.W, ir.P, ir.Q, ir.stride, ir.f16)) return false;
  // the output must not land on anything the block reads: tiles read beyond their own pixels
  const uintptr_t olo = (uintptr_t)c.out;
  const size_t obytes = (size_t)g.N * g.K * g.P * g.Q * 2;
  bool clash = false;
  for (const ConvJob *j : job)
    for (int k = 0; k < 3; ++k) clash = clash || ranges_overlap(olo, olo + obytes, j->dep_lo[k], j->dep_hi[k]);
  void *dst = clash ? home_acquire(obytes) : c.out;
  if (!dst) return false;
  ir.y = (bf16 *)dst;
  if (!launch_ir(ir, r.stream)) return false;
  mark_act16(c.out, g.N, g.K, g.P, g.Q, clash ? dst : nullptr);
  return true;
}

// Makes the sum of two held-back convolutions one kernel's: `b` takes `a` along.  False when no kernel does, or one of
// the operands is not there to stay.
bool join_summands(const ConvJob &a, ConvJob &b) {
  auto plain = [](const TcConvArgs &t) {
    return t.R == 1 && t.S == 1 && t.pad_h == 0 && t.pad_w == 0 && !t.w_step;
  };
  auto strided = [](const TcConvArgs &t) { return t.stride_h != 1 || t.stride_w != 1; };
  // the second summand is a 1x1 convolution, the strided one of two
  const bool swap = plain(a.a) && (!plain(b.a) || (strided(a.a) && !strided(b.a)));
  const TcConvArgs &first = swap ? b.a : a.a, &second = swap ? a.a : b.a;
  if (!plain(second)) return false;
  TcConvArgs c = first;
  c.x2 = second.x; c.w2 = second.w; c.bias2 = second.bias;
  c.H2 = second.H; c.W2 = second.W; c.Cf2 = second.Cf;
  c.stride2_h = second.stride_h; c.stride2_w = second.stride_w;
  c.consts_ready = a.a.consts_ready && b.a.consts_ready;
  c.y = b.a.y;
  if (!tc_conv_supported(c)) return false;
  b.a = c;
  b.dep_lo[3] = a.dep_lo[0]; b.dep_hi[3] = a.dep_hi[0];
  b.dep_lo[4] = a.dep_lo[2]; b.dep_hi[4] = a.dep_hi[2];
  return true;
}

// The other summand by itself: no kernel takes both.
void launch_summand() {
  if (!g_pending.after_summand) return;
  g_pending.after_summand = false;
  launch_job(g_front[0]);
  g_fronts = 0;
}

// A convolution and the one behind it that reads its result as one kernel; false when they have to run one by one.
bool launch_two(ConvJob &a, ConvJob &b) {
  a.a.act = a.g.act;
  b.a.act = b.g.act;
  if (a.depthwise || b.depthwise || a.product || b.product || !tc_pair_supported(a.a, b.a)) return false;
  const size_t ybytes = (size_t)a.g.N * a.g.K * a.g.P * a.g.Q * 2, tbytes = (size_t)b.g.N * b.g.K * b.g.P * b.g.Q * 2;
  // neither result may land on what other tiles have still to read; the shortcut tensor's place, exactly, is
  // as good as any (each tile reads its part before it stores)
  auto clash = [&](const void *p, size_t bytes, const ConvJob &j, bool in_place_ok) {
    const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
    for (int k = 0; k < 5; ++k)
      if (ranges_overlap(lo, hi, j.dep_lo[k], j.dep_hi[k]) &&
          !(in_place_ok && k == 1 && lo == j.dep_lo[k] && hi == j.dep_hi[k]))
        return true;
    return false;
  };
  void *y = a.out, *t = b.out;
  if (clash(y, ybytes, a, true) || clash(y, ybytes, b, false)) y = home_acquire(ybytes);
  if (!y) return false;
  a.a.y = (bf16 *)y;
  const uintptr_t ylo = (uintptr_t)y;
  if (clash(t, tbytes, a, false) || clash(t, tbytes, b, false) ||
      ranges_overlap((uintptr_t)t, (uintptr_t)t + tbytes, ylo, ylo + ybytes))
    t = home_acquire(tbytes);
  if (!t) return false;
  b.a.y = (bf16 *)t;
  b.a.x = nullptr;
  if (!launch_tc_pair(a.a, b.a, rt().stream)) return false;
  mark_act16(a.out, a.g.N, a.g.K, a.g.P, a.g.Q, y == a.out ? nullptr : y);
  mark_act16(b.out, b.g.N, b.g.K, b.g.P, b.g.Q, t == b.out ? nullptr : t);
  return true;
}

// Executes the held-back convolution as far as it has been built up.
void flush_pending() {
  if (!g_pending.active) return;
  g_pending.active = false;
  for (int i = 0; i < g_fronts; ++i)
    if (g_front[i].absorbed) trace_count_chain();
  if (g_pending.absorbed && !g_pending.product) trace_count_chain();   // convolution chains
  launch_summand();
  if (g_pending.follows) {
    g_pending.follows = false;
    ConvJob &lead = g_front[0];
    if (!launch_two(lead, g_pending)) {
      launch_job(lead);
      g_pending.a.x = act16_ptr(lead.out);
      if ((const void *)g_pending.a.x == lead.out) {
        g_pending.dep_lo[0] = (uintptr_t)lead.out;
        g_pending.dep_hi[0] = (uintptr_t)lead.out + (size_t)lead.g.N * lead.g.K * lead.g.P * lead.g.Q * 2;
      }
      launch_job(g_pending);
    }
    g_fronts = 0;
    return;
  }
  if (g_fronts != 2 || !launch_block(g_front[0], g_front[1], g_pending)) {
    const bf16 *x = nullptr;
    auto resolve = [&](ConvJob &job) {
      const ConvGeom &g = job.g;
      if (job.joined) (job.depthwise ? job.dw_x : job.a.x) = x;
      if ((job.linked || job.joined) && !job.depthwise && job.a.Cf != g.C) {
        bf16 *xp = (bf16 *)scratch_get(6, (size_t)g.N * job.a.Cf * g.H * g.W * 2);
        launch_pad_channels_bf16(job.a.x, xp, (int64_t)g.N * g.H * g.W, g.C, job.a.Cf, rt().stream);
        job.a.x = xp;
        job.dep_lo[0] = job.dep_hi[0] = 0;
      }
    };
    for (int i = 0; i < g_fronts; ++i) {
      resolve(g_front[i]);
      x = launch_job(g_front[i], true);
    }
    resolve(g_pending);
    launch_job(g_pending);
  }
  g_fronts = 0;
}

// [p, p+bytes) is about to be overwritten or freed (`writes`), or merely handed out again:
// in the first case whatever still has to read it must run first.  Handing a range out
// writes nothing (its zero fill is lazy), so a held-back convolution may keep reading its
// inputs from it; launch_job() deals with the case that its own output lands there.
void pending_guard_range(const void *p, size_t bytes, bool writes) {
  if (!g_pending.active) return;
  const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
  if (writes)
    for (int j = 0; j <= g_fronts; ++j) {
      const ConvJob &job = j < g_fronts ? g_front[j] : g_pending;
      for (int k = 0; k < 5; ++k)
        if (ranges_overlap(lo, hi, job.dep_lo[k], job.dep_hi[k])) {
          if (rt().log) fprintf(stderr, "[occamy] held-back conv runs early: input %d overwritten\n", k);
          flush_pending();
          return;
        }
    }
  // the tensor it is going to write must also still belong to it
  auto takes_output = [&](const ConvJob &job) {
    const uintptr_t olo = (uintptr_t)job.out;
    const size_t elem = job.a.split || job.product ? 4 : 2;
    return ranges_overlap(lo, hi, olo, olo + (size_t)job.g.N * job.g.K * job.g.P * job.g.Q * elem);
  };
  if (takes_output(g_pending) || ((g_pending.after_summand || g_pending.follows) && takes_output(g_front[0]))) {
    if (rt().log) fprintf(stderr, "[occamy] held-back conv runs early: output re-handed out\n");
    flush_pending();
  }
}

// Common tail of every traced entry point: record the call, end the speculation when the
// recorded sequence is left, run the held-back convolution unless this call continues it.
void before_write_hook(const void *p, size_t bytes) { pending_guard_range(p, bytes, true); }

Role step(Entry &e, bool passive) {
  rt().before_write = before_write_hook;
  rt().home_held = home_held_hook;
  if (graph_covers(e)) return R_SKIP;
  graph_uncovered();
  bool deviated = false;
  const Role role = trace_step(e, &deviated);
  if (deviated) {
    graph_left_recording();
    graph_stop_capture();
    g_pending.out16 = false;   // who reads it is not known any more
    g_pending.out_parts = g_pending.a.split && g_pending.res_set;
    flush_pending();
    settle_sources();   // nor who reads the inputs: back to their plain form
    // Tensors that fusion skipped earlier in this inference stay unwritten.  The recorded
    // program had no reader for them; should this (different) program read one, that read
    // reports error 990.  A shared prefix alone - two models with the same first layers - is
    // not an error.
    if (trace_has_elided() && rt().log)
      fprintf(stderr, "[occamy] call sequence left the recorded one after tensors were skipped\n");
  }
  if (!passive && role != R_ABSORB && !((trace_last_flags() & RF_JOIN) && g_pending.active && g_pending.linked) &&
      !((trace_last_flags() & RF_SUM) && g_pending.active && g_pending.summand) &&
      !((trace_last_flags() & RF_FOLLOW) && g_pending.active && g_pending.leads)) {
    if (g_pending.active && rt().log)
      fprintf(stderr, "[occamy] held-back conv closed by call sym %d (absorbed %d)\n", e.sym,
              g_pending.absorbed);
    flush_pending();
  }
  return role;
}

// A call's arguments in its trace entry (run_again makes the call from them).
void put(Entry &e, std::initializer_list<const void *> ptrs) {
  int i = 0;
  for (const void *p : ptrs) e.args.p[i++] = const_cast<void *>(p);
}
// appends n values behind the ones already there
void put(Entry &e, int &at, const int64_t *d, int64_t n) {
  if (n > 24 - at) e.args.whole = false;
  for (int64_t i = 0; i < n && at < 24; ++i) e.args.v[at++] = d[i];
}
void put(Entry &e, int &at, int64_t v) { put(e, at, &v, 1); }

// A device-to-device copy into tensor `rec` whose readers are convolutions of the 16-bit path: brings it in
// in the form they take, straight from the source (the plain copy and the conversion behind it moved
// the batch twice: 79 us of a batch-256 ResNet-50).  False when the form is not known, or when the source is a
// tensor of the runtime's, whose memory later calls may write.
bool copy_for_conv(const float *src, float *dst, size_t bytes, TensorRec *rec) {
  Runtime &r = rt();
  const Entry *rd = (trace_last_flags() & RF_FOR_CONV) ? trace_last_reader() : nullptr;
  if (!rd || r.mode == MATH_FP32 || reg_find(src)) return false;
  const int64_t *v = rd->args.v;   // dX[4], dW[4], pads[2], strides[2], groups
  ConvGeom g;
  memset(&g, 0, sizeof(g));
  g.N = (int)v[0]; g.C = (int)v[1]; g.H = (int)v[2]; g.W = (int)v[3];
  g.R = (int)v[6]; g.S = (int)v[7];
  g.pad_w = (int)v[9]; g.stride_w = (int)v[11];
  if ((size_t)numel4(v) * 4 != bytes) return false;
  void *home;
  if (g.C >= 16) {
    home = home_acquire(bytes / 2);
    if (!home) return false;
    launch_nchw_f32_to_nhwc_bf16(src, (bf16 *)home, g.N, g.C, g.H, g.W, mode_f16(), r.stream);
    mark_act16(dst, g.N, g.C, g.H, g.W, home);
  } else {
    if (v[12] != 1) return false;
    g.Q = (g.W + 2 * g.pad_w - g.S) / g.stride_w + 1;
    int Cp, Sp, Wp;
    stem_geometry(g, Cp, Sp, Wp);
    home = home_acquire((size_t)g.N * g.H * Wp * Cp * 2);
    if (!home) return false;
    launch_pad_input_bf16(src, (bf16 *)home, g.N, g.C, g.H, g.W, Wp, Cp, g.pad_w, mode_f16(), r.stream);
    rec->fmt = FMT_STEM_ROWS;
    rec->n = g.N; rec->c = g.C; rec->h = g.H; rec->w = g.W;
    rec->home = home;
    rec->stem_wp = Wp; rec->stem_cp = Cp; rec->stem_pad = g.pad_w; rec->stem_f16 = mode_f16();
    rec->host_src = nullptr;
  }
  rec->dev_src = src;
  return true;
}

// Opens every traced entry point: when the call has been carried out, a recorded stretch of calls
// may begin or end behind it.
struct CallScope {
  ~CallScope() { graph_after_call(); }
};

void elide(void *p) {
  uintptr_t base;
  TensorRec *rec = reg_find(p, &base);
  if (rec && base == (uintptr_t)p) rec->fmt = FMT_ELIDED;
  trace_note_elided();
}

// Geometry of a convolution call; false when its shapes do not fit together.
bool conv_geometry(const int64_t *dX, const int64_t *dW, int64_t groups, const int64_t *pads, const int64_t *strides,
                   int act, float lo, float hi, ConvGeom &g) {
  g.N = (int)dX[0]; g.C = (int)dX[1]; g.H = (int)dX[2]; g.W = (int)dX[3];
  g.K = (int)dW[0]; g.R = (int)dW[2]; g.S = (int)dW[3];
  g.groups = (int)(groups < 1 ? 1 : groups);
  g.pad_h = (int)pads[0]; g.pad_w = (int)pads[1];
  g.stride_h = (int)strides[0]; g.stride_w = (int)strides[1];
  g.act = act; g.lo = lo; g.hi = hi;
  const bool shape_ok = !(g.stride_h < 1 || g.stride_w < 1 || g.C % g.groups || g.K % g.groups ||
                          dW[1] * g.groups != g.C);
  g.P = shape_ok ? (g.H + 2 * g.pad_h - g.R) / g.stride_h + 1 : 0;
  g.Q = shape_ok ? (g.W + 2 * g.pad_w - g.S) / g.stride_w + 1 : 0;
  return shape_ok;
}

// Activation of the fused convolution call's mode; mode 3 is ReLU6.
int act_of_mode(int64_t mode, float &lo, float &hi) {
  lo = 0.f;
  hi = mode == 3 ? 6.f : 0.f;
  return mode == 1 ? ACT_RELU : mode == 3 ? ACT_CLIP : mode == 0 ? ACT_SIGMOID : mode == 2 ? ACT_TANH : ACT_IDENTITY;
}

float *conv_common(int sym, float *x, const int64_t *dX, float *w, const int64_t *dW, float *bias,
                   int64_t groups, const int64_t *pads, const int64_t *strides, int64_t act_mode, float *y) {
  Runtime &r = rt();
  ConvGeom g;
  float lo, hi;
  const int act = act_of_mode(act_mode, lo, hi);
  const bool shape_ok = conv_geometry(dX, dW, groups, pads, strides, act, lo, hi, g);
  const bool depthwise = g.groups > 1 && g.groups == g.C && g.K == g.C;

  CallScope scope;
  Entry e = trace_entry(sym);
  int at = 0;
  put(e, {x, w, bias, y});
  put(e, at, dX, 4); put(e, at, dW, 4); put(e, at, pads, 2); put(e, at, strides, 2);
  put(e, at, groups); put(e, at, act_mode);
  te_ptr(e, x); te_ptr(e, w); te_ptr(e, bias); te_ptr(e, y);
  te_dims(e, dX, 4); te_dims(e, dW, 4); te_dims(e, pads, 2); te_dims(e, strides, 2);
  te_i(e, groups); te_i(e, act_mode);
  e.in[0] = (uintptr_t)x; e.in[1] = (uintptr_t)w; e.in[2] = (uintptr_t)bias;
  e.in_bytes[0] = numel4(dX) * 4; e.in_bytes[1] = numel4(dW) * 4; e.in_bytes[2] = dW[0] * 4;
  e.out = (uintptr_t)y;
  e.dims[0] = g.N; e.dims[1] = g.K; e.dims[2] = g.P; e.dims[3] = g.Q;
  e.out_bytes = (int64_t)g.N * g.K * g.P * g.Q * 4;
  e.kind = (int)act_mode;
  e.depthwise = depthwise;
  e.fusable = shape_ok && r.mode != MATH_FP32 && g.P > 0 && g.Q > 0 && g.N > 0 &&
              (depthwise ? g.C % 8 == 0
                         : (g.groups == 1 && g.K % 8 == 0 && (g.C < 16 || g.C % 8 == 0)));
  e.parts = shape_ok && r.mode == MATH_FP32 && g.P > 0 && g.Q > 0 && g.N > 0 && !depthwise && parts_shape_ok(g);
  e.fusable = e.fusable || e.parts;
  // the fused convolution + max-pool kernel takes 64-channel stems whose column step is 16 bytes
  e.poolable = e.fusable && r.mode == MATH_BF16 && !depthwise && g.C <= 4 && g.K == 64 && g.stride_w == 2 && g.Q <= 128 &&
               g.S <= 16 && g.R <= 11;
  const Role role = step(e, false);
  if (role == R_SKIP) return y;
  const uint16_t flags = trace_last_flags();
  bool join = false, sum = false, follow = false;
  if (g_pending.active && g_pending.leads) {   // left by step(): this call was recorded as reading its result
    const ConvGeom &f = g_pending.g;
    follow = role == R_DEFER && e.fusable && !e.parts && !depthwise && stays_packed(w) && !g_fronts && g_pending.out == x &&
             f.N == g.N && f.K == g.C && f.P == g.H && f.Q == g.W && g.C % 16 == 0;
    if (!follow) flush_pending();
  } else if (g_pending.active && g_pending.summand) {   // left by step(): this call was recorded as the other summand
    const ConvGeom &f = g_pending.g;
    sum = role == R_DEFER && e.fusable && !depthwise && !e.parts && f.N == g.N && f.K == g.K &&
          f.P == g.P && f.Q == g.Q && !g_pending.act_set && !g_pending.res_set;
    if (!sum) flush_pending();
  } else if (g_pending.active) {   // left by step() because this call was recorded as joining it
    const ConvGeom &f = g_pending.g;
    join = role == R_DEFER && e.fusable && !e.parts && stays_packed(w) && g_fronts < 2 && g_pending.out == x && f.N == g.N && f.K == g.C &&
           f.P == g.H && f.Q == g.W && (depthwise ? g_fronts == 0 : g_fronts == 1 && g.C % 16 == 0);
    if (!join) flush_pending();
  }

  if (!shape_ok) {
    set_error(997, "convolution: inconsistent shape");
    return y;
  }
  if (g.P <= 0 || g.Q <= 0 || g.N == 0) return y;
  if (r.log)
    fprintf(stderr, "[occamy] conv x[%d,%d,%d,%d] w[%d,%d,%d,%d] g%d s%d p%d act%d role%d\n", g.N,
            g.C, g.H, g.W, g.K, (int)dW[1], g.R, g.S, g.groups, g.stride_h, g.pad_h, act,
            (int)role);
  // One of two summands, prepared: the second finds the first held back (unless an upload had to run it), the first
  // may wait for it when its operands stay where they are.
  auto hold_summand = [&](ConvJob &job, bool in_place) {
    if (sum && g_pending.active) {
      g_front[0] = g_pending;
      g_fronts = 1;
      job.after_summand = true;
    } else if (!sum) {
      job.summand = role == R_DEFER && (flags & RF_SUM) && !depthwise && in_place && stays_packed(w);
    }
  };
  if (r.mode != MATH_FP32) {
    ConvJob job;
    // (the first of three takes its input as it is)
    job.linked = role == R_DEFER && (flags & RF_LINK) && stays_packed(w) && (join || (!(flags & RF_JOIN) && is_act16(x, g.N, g.C, g.H, g.W)));
    job.joined = join || follow;
    job.leads = role == R_DEFER && (flags & RF_LEAD) && !depthwise && stays_packed(w);
    bool ok = depthwise ? prepare_depthwise(x, w, bias, g, job)
                        : (g.groups == 1 && prepare_dense(x, w, bias, g, job));
    if (follow && ok && g_pending.active) {
      g_front[0] = g_pending;
      g_fronts = 1;
      job.joined = false;
      job.follows = true;
    } else if (follow) {   // (an upload had to run it, or this one is not taken)
      flush_pending();
      job = ConvJob();
      ok = prepare_dense(x, w, bias, g, job);
    } else if (join && ok && g_pending.active) {
      // nothing else reads what the one in front would have written
      g_front[g_fronts++] = g_pending;
      elide(g_pending.out);
    } else if (join) {
      // cannot be carried on with, or a constant's upload was about to overwrite something the ones in
      // front still had to read, and they have run
      flush_pending();
      job = ConvJob();
      ok = depthwise ? prepare_depthwise(x, w, bias, g, job) : prepare_dense(x, w, bias, g, job);
    }
    if (ok) {
      job.out = y;
      hold_summand(job, is_act16(x, g.N, g.C, g.H, g.W) && g.C % 16 == 0);
      if (role == R_DEFER) {   // later calls of the recorded sequence fold into this one
        if (e.poolable && !depthwise && job.a.w_step) {
          // the pool that may join later runs after the filter tensor has been given back
          const int cp = job.a.w_step / g.stride_w;
          job.w_stem = (const bf16 *)packed_weights(w, PACK_STEM, stem_pool_weight_bytes(g.R, job.a.Cf),
                                                    g.K, g.C, g.R, g.S, job.a.Cf / cp, cp);
        }
        g_pending = job;
        g_pending.active = true;
        return y;
      }
      launch_job(job);
      return y;
    }
  }
  if (e.parts) {
    ConvJob job;
    job.out = y;
    if (prepare_parts(x, w, bias, g, job)) {
      job.out_parts = (flags & RF_FOR_PARTS) && g.K % 16 == 0;
      if (role == R_DEFER) {
        g_pending = job;
        g_pending.active = true;
      } else {
        launch_job(job);
      }
      return y;
    }
  }
  flush_pending();   // (a summand that this convolution does not go with after all)
  ensure_f32(x);
  const float *wd = operand_f32(w, (size_t)numel4(dW) * 4);
  const float *bd = bias ? operand_f32(bias, (size_t)g.K * 4) : nullptr;
  if (depthwise) launch_depthwise_f32(x, wd, bd, y, g, r.stream);
  else launch_conv_f32(x, wd, bd, y, g, r.stream);
  mark_f32(y);
  return y;
}

// The held-back convolution takes over a following element-wise call.  `out` is where that
// call would have written; the convolution's own output is skipped unless it is the same.
void pending_retarget(float *out) {
  g_pending.absorbed++;
  if (out != g_pending.out) {
    elide(g_pending.out);
    g_pending.out = out;
  }
  // (a residual exists in planes only, and only such results can take one along)
  g_pending.out_parts = g_pending.a.split && !g_pending.product && g_pending.g.K % 16 == 0 &&
                        (g_pending.res_set || (trace_last_flags() & RF_FOR_PARTS));
}

int64_t prod(const int64_t *d, int64_t rank) {
  int64_t n = 1;
  for (int64_t i = 0; i < rank; ++i) n *= d[i];
  return n;
}

}  // namespace

extern "C" {

// ---------------------------------------------------------------- memory pool
cudaError_t wrapDNNMalloc(void **devPtr, size_t size) {
  rt();
  cudaError_t err = device_malloc(devPtr, size ? size : 1);
  if (err != cudaSuccess) die("Malloc", err, size);
  CallScope scope;
  Entry e = trace_entry(S_MALLOC);
  te_i(e, (int64_t)size);
  e.out = (uintptr_t)*devPtr;
  e.out_bytes = (int64_t)size;
  step(e, true);
  pending_guard_range(*devPtr, size, false);
  reg_new(*devPtr, size, FMT_ZERO);  // zero fill is issued only if somebody reads it unwritten
  return cudaSuccess;
}

cudaError_t wrapDNNMemPoolInit(void **devPtr, size_t size) {
  Runtime &r = rt();
  *devPtr = nullptr;
  cudaEvent_t ready = nullptr;
  int same = 0;
  for (const CachedPool &c : g_pool_cache) same += c.bytes == size;
  if (same >= pool_cache_blocks() && same > 0) {
    for (size_t i = 0; i < g_pool_cache.size(); ++i)   // the oldest block of this size
      if (g_pool_cache[i].bytes == size) {
        *devPtr = g_pool_cache[i].base;
        ready = g_pool_cache[i].done;
        g_pool_cache.erase(g_pool_cache.begin() + i);
        break;
      }
  } else {
    // blocks of other sizes make room first
    for (size_t i = 0; i < g_pool_cache.size();)
      if (g_pool_cache[i].bytes != size) {
        free_cached_pool(g_pool_cache[i]);
        g_pool_cache.erase(g_pool_cache.begin() + i);
      } else {
        ++i;
      }
    cudaError_t err = device_malloc(devPtr, size ? size : 1);
    if (err != cudaSuccess && !g_pool_cache.empty()) {   // no room for a second block
      *devPtr = g_pool_cache[0].base;
      ready = g_pool_cache[0].done;
      g_pool_cache.erase(g_pool_cache.begin());
    } else if (err != cudaSuccess) {
      die("MemPoolInit", err, size);
    }
  }
  if (g_block_ready) OCC_CUDA(cudaEventDestroy(g_block_ready));
  g_block_ready = ready;
  g_cur_pool = *devPtr;
  g_cur_pool_bytes = size;
  g_launches_at_pool_init = r.counters[CNT_LAUNCHES] + r.main_copies;
  g_pools.push_back(PoolRec{*devPtr, size});
  if ((int64_t)size > r.counters[CNT_POOL_HWM]) r.counters[CNT_POOL_HWM] = (int64_t)size;
  trace_set_pool(*devPtr, size);
  CallScope scope;
  Entry e = trace_entry(S_POOLINIT);
  te_i(e, (int64_t)size);
  step(e, false);
  return cudaSuccess;
}

static void hand_out(void *p, size_t bytes) {
  CallScope scope;
  Entry e = trace_entry(S_MEMOFFSET);
  te_ptr(e, p);
  te_i(e, (int64_t)bytes);
  e.out = (uintptr_t)p;
  e.out_bytes = (int64_t)bytes;
  put(e, {p});
  e.args.v[0] = (int64_t)bytes;
  if (step(e, true) == R_SKIP) return;
  pending_guard_range(p, bytes, false);
  reg_new(p, bytes, FMT_ZERO);
}

cudaError_t wrapDNNMemOffset(void **devPtr, void *basePtr, size_t offset, size_t mallocSize) {
  *devPtr = (char *)basePtr + offset;
  hand_out(*devPtr, mallocSize);
  return cudaSuccess;
}

cudaError_t wrapDNNMemcpy(void *dst, const void *src, size_t count_, int kind,
                          cudaStream_t /*stream*/) {
  Runtime &r = rt();
  if (count_ == 0) return cudaSuccess;
  cudaError_t err = cudaSuccess;
  CallScope scope;
  if (kind == 1 || kind == 3) {
    Entry e = trace_entry(kind == 1 ? S_H2D : S_D2D);
    if (kind == 1) te_ptr(e, dst);
    else te_ptr_or_elsewhere(e, dst);
    te_i(e, (int64_t)count_);
    put(e, {dst});
    e.args.v[0] = (int64_t)count_;
    uint64_t hash = 0;
    if (kind == 1) {
      hash = host_hash(src, count_);
      e.args.v[1] = (int64_t)hash;
      e.host = src;
    }
    if (kind == 3) {
      te_ptr_or_elsewhere(e, src);
      e.in[0] = (uintptr_t)src;
      e.in_bytes[0] = (int64_t)count_;
    }
    e.out = (uintptr_t)dst;
    e.out_bytes = (int64_t)count_;
    if (step(e, kind == 1) == R_SKIP) return cudaSuccess;
    uintptr_t base;
    if (kind == 3) {
      pending_guard_range(dst, count_, true);
      const TensorRec *from = reg_find(src, &base);
      if (from && base == (uintptr_t)src && fmt_is_16(from->fmt) && !reg_find(dst) &&
          (size_t)(from->n * from->c * from->h * from->w) * 4 == count_) {
        // a 16-bit result on its way out: converted straight into the caller's memory
        launch_nhwc_bf16_to_nchw_f32(act16_ptr(src), (float *)dst, (int)from->n, (int)from->c, (int)from->h,
                                     (int)from->w, from->fmt == FMT_F16_NHWC, r.stream);
        count(CNT_MATERIALIZE);
        return cudaSuccess;
      }
      ensure_f32(src);
    }
    TensorRec *rec = reg_find(dst, &base);
    const bool whole = rec && base == (uintptr_t)dst && count_ + 32 > rec->bytes;
    if (kind == 3 && whole && copy_for_conv((const float *)src, (float *)dst, count_, rec)) return cudaSuccess;
    if (rec && !whole) ensure_f32(dst);
    if (kind == 1 && whole) {
      rec->host_src = src;
      rec->host_bytes = count_;
      rec->host_hash = hash;
      // A constant whose packed form is already resident need not cross PCIe again; the
      // copy is made later only if something other than a convolution / GEMM reads it.
      if (r.cache_weights) {
        auto it = r.resident.find(src);
        if (it != r.resident.end() && it->second.first == count_ &&
            it->second.second == rec->host_hash) {
          rec->fmt = FMT_PENDING;   // nothing is written now
          count(CNT_H2D_SKIPPED, (int64_t)count_);
          return cudaSuccess;
        }
      }
    }
    if (kind == 1) {
      graph_before_upload();
      trace_mark_uploaded();
      pending_guard_range(dst, count_, true);
    }
    const bool in_pool = g_cur_pool && (uintptr_t)dst >= (uintptr_t)g_cur_pool &&
                         (uintptr_t)dst + count_ <= (uintptr_t)g_cur_pool + g_cur_pool_bytes;
    if (kind == 1 && whole && in_pool && count_ >= (1u << 20) && pool_cache_blocks() >= 2) {
      // Large upload into a fresh tensor of this inference's pool block: nothing enqueued
      // for this inference touches these bytes yet, and the block's previous user is done
      // once `g_block_ready` has fired, so the copy need not queue behind the kernels of
      // the previous inference.  Later work on the launch stream waits for it.
      if (!g_copy_stream) OCC_CUDA(cudaStreamCreateWithFlags(&g_copy_stream, cudaStreamNonBlocking));
      if (g_block_ready) OCC_CUDA(cudaStreamWaitEvent(g_copy_stream, g_block_ready, 0));
      if (r.counters[CNT_LAUNCHES] + r.main_copies != g_launches_at_pool_init) {
        // work of this inference is already queued and may still read bytes that the pool
        // plan has recycled for this tensor: the copy goes behind it
        cudaEvent_t before;
        OCC_CUDA(cudaEventCreateWithFlags(&before, cudaEventDisableTiming));
        OCC_CUDA(cudaEventRecord(before, r.stream));
        OCC_CUDA(cudaStreamWaitEvent(g_copy_stream, before, 0));
        OCC_CUDA(cudaEventDestroy(before));
      }
      if (graph_upload_in_pieces(dst, src, count_, g_copy_stream)) {
        count(CNT_H2D_BYTES, (int64_t)count_);
        rec->fmt = FMT_F32;
        rec->home = rec->dev_src = nullptr;
        return cudaSuccess;
      }
      err = cudaMemcpyAsync(dst, src, count_, cudaMemcpyHostToDevice, g_copy_stream);
      cudaEvent_t ev;
      OCC_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      OCC_CUDA(cudaEventRecord(ev, g_copy_stream));
      OCC_CUDA(cudaStreamWaitEvent(r.stream, ev, 0));
      OCC_CUDA(cudaEventDestroy(ev));
    } else {
      err = cudaMemcpyAsync(dst, src, count_,
                            kind == 1 ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice,
                            r.stream);
      r.main_copies++;
    }
    if (kind == 1) count(CNT_H2D_BYTES, (int64_t)count_);
    if (rec && whole) {
      rec->fmt = FMT_F32;
      rec->home = rec->dev_src = nullptr;
      if (kind == 3) rec->host_src = nullptr;
    }
  } else if (kind == 2) {
    Entry e = trace_entry(S_D2H);
    te_ptr(e, src);
    te_i(e, (int64_t)count_);
    e.in[0] = (uintptr_t)src;
    e.in_bytes[0] = (int64_t)count_;
    step(e, false);
    settle_sources();   // (the call waits for the stream)
    uintptr_t base;
    TensorRec *rec = reg_find(src, &base);
    const void *from = src;
    if (rec && fmt_is_16(rec->fmt) && base == (uintptr_t)src) {
      // convert into scratch instead of in place: the tensor keeps its fast format
      const size_t elems = (size_t)(rec->n * rec->c * rec->h * rec->w);
      float *tmp = (float *)scratch_get(2, elems * 4);
      launch_nhwc_bf16_to_nchw_f32(act16_ptr(src), tmp, (int)rec->n, (int)rec->c, (int)rec->h,
                                   (int)rec->w, rec->fmt == FMT_F16_NHWC, r.stream);
      count(CNT_MATERIALIZE);
      from = tmp;
    } else {
      ensure_f32(src);
    }
    // Small results go through a pinned buffer: one transfer the driver need not stage.
    if (count_ <= STAGE_BYTES && !r.host_stage) {
      if (cudaMallocHost(&r.host_stage, STAGE_BYTES) != cudaSuccess) cudaGetLastError();
    }
    void *to = count_ <= STAGE_BYTES && r.host_stage ? r.host_stage : dst;
    err = cudaMemcpyAsync(to, from, count_, cudaMemcpyDeviceToHost, r.stream);
    if (err == cudaSuccess) err = cudaStreamSynchronize(r.stream);
    if (err == cudaSuccess && to != dst) memcpy(dst, to, count_);
    poll_watchdog();
  } else {
    Entry e = trace_entry(S_OPAQUE);
    step(e, false);
    settle_sources();
    err = cudaMemcpyAsync(dst, src, count_, (cudaMemcpyKind)kind, r.stream);
    if (err == cudaSuccess) err = cudaStreamSynchronize(r.stream);
  }
  if (err != cudaSuccess) {
    printf("[Memcpy] GPU error: %s\n", cudaGetErrorString(err));
    exit(-1);
  }
  return cudaSuccess;
}

cudaError_t wrapDNNDealloc(void *devPtr) {
  Runtime &r = rt();
  if (!devPtr) return cudaSuccess;
  size_t bytes = 0;
  bool was_pool = false;
  for (size_t i = 0; i < g_pools.size(); ++i)
    if (g_pools[i].base == devPtr) {
      bytes = g_pools[i].bytes;
      was_pool = true;
      g_pools.erase(g_pools.begin() + i);
      break;
    }
  CallScope scope;
  if (was_pool) {
    Entry e = trace_entry(S_POOLFREE);
    step(e, false);   // runs whatever is still held back
    trace_set_pool(nullptr, 0);
    if (devPtr == g_cur_pool) {
      g_cur_pool = nullptr;
      g_cur_pool_bytes = 0;
    }
    if (pool_cache_blocks() > 0) {
      // Work still in flight on the launch stream is ordered before anything a later
      // inference enqueues there, so the block can be handed out again without waiting;
      // the event lets the copy stream know when its bytes are really free.
      if (bytes) reg_drop_range(devPtr, bytes);
      CachedPool c{devPtr, bytes, nullptr};
      OCC_CUDA(cudaEventCreateWithFlags(&c.done, cudaEventDisableTiming));
      OCC_CUDA(cudaEventRecord(c.done, r.stream));
      g_pool_cache.push_back(c);
      while ((int)g_pool_cache.size() > pool_cache_blocks()) {
        free_cached_pool(g_pool_cache[0]);
        g_pool_cache.erase(g_pool_cache.begin());
      }
      return cudaSuccess;
    }
  } else {
    uintptr_t base;
    TensorRec *rec = reg_find(devPtr, &base);
    if (rec && base == (uintptr_t)devPtr) bytes = rec->bytes;
    Entry e = trace_entry(S_DEALLOC);
    te_ptr(e, devPtr);
    e.out = (uintptr_t)devPtr;
    e.out_bytes = (int64_t)bytes;
    step(e, true);
    pending_guard_range(devPtr, bytes ? bytes : 1, true);
  }
  settle_sources();
  OCC_CUDA(cudaStreamSynchronize(r.stream));
  if (bytes) reg_drop_range(devPtr, bytes);
  cudaError_t err = cudaFree(devPtr);
  if (err != cudaSuccess) {
    printf("[Dealloc] GPU error: %s\n", cudaGetErrorString(err));
    exit(-1);
  }
  return cudaSuccess;
}

// ---------------------------------------------------------------- handle
// The compiled function creates the handle on entry and destroys it before it returns:
// these two calls delimit one inference for the call trace.
int cudnnCreate(cudnnContext **handle) {
  rt();
  *handle = reinterpret_cast<cudnnContext *>(malloc(16));
  graph_inference_begin();
  went_forwards();   // (whatever brought the input in)
  flush_pending();
  trace_begin();
  return *handle ? 0 : 2;
}
int cudnnDestroy(cudnnContext *handle) {
  graph_inference_end();
  flush_pending();
  trace_end();
  free(handle);
  return 0;
}

// ---------------------------------------------------------------- convolution
float *DNNConvFunc(cudnnContext *, float *x, int64_t dimX[4], float *w, int64_t dimW[4],
                   float * /*workspace*/, int64_t /*workspaceSize*/, int64_t /*algo*/,
                   int64_t groups, int64_t pads[2], int64_t strides[2], float *y) {
  return conv_common(S_CONV, x, dimX, w, dimW, nullptr, groups, pads, strides, 5, y);
}

float *DNNConvBiasActivFunc(cudnnContext *, float *x, int64_t dimX[4], float *w, int64_t dimW[4],
                            float *bias, int64_t dimB[4], float * /*workspace*/,
                            int64_t /*workspaceSize*/, int64_t /*algo*/, int64_t pads[2],
                            int64_t strides[2], int64_t activMode, float *y) {
  (void)dimB;
  return conv_common(S_CONV_BIAS_ACT, x, dimX, w, dimW, bias, 1, pads, strides, activMode, y);
}

// ---------------------------------------------------------------- element-wise
float *DNNActiveFunc(cudnnContext *, float *x, int64_t dimX[4], int32_t mode, float *y) {
  Runtime &r = rt();
  const int64_t n = numel4(dimX);
  const int act = mode == 0 ? ACT_SIGMOID : (mode == 1 ? ACT_RELU : (mode == 2 ? ACT_TANH : ACT_IDENTITY));
  CallScope scope;
  Entry e = trace_entry(S_ACTIVE);
  int at = 0;
  put(e, {x, y});
  put(e, at, dimX, 4); put(e, at, mode);
  te_ptr(e, x); te_ptr(e, y); te_dims(e, dimX, 4); te_i(e, mode);
  e.in[0] = (uintptr_t)x; e.in_bytes[0] = n * 4; e.out = (uintptr_t)y; e.out_bytes = n * 4;
  for (int i = 0; i < 4; ++i) e.dims[i] = dimX[i];
  e.kind = mode == 1 ? CK_RELU : CK_NONE;
  const Role role = step(e, false);
  if (role == R_SKIP) return y;
  if (role == R_ABSORB && g_pending.active) {
    const ConvGeom &g = g_pending.g;
    if (mode == 1 && x == g_pending.out && !g_pending.act_set && dimX[0] == g.N &&
        dimX[1] == g.K && dimX[2] == g.P && dimX[3] == g.Q) {
      pending_retarget(y);
      g_pending.g.act = ACT_RELU;
      g_pending.act_set = true;
      if (!g_pending.linked && !g_pending.leads) flush_pending();   // an activation closes the chain
      return y;
    }
    flush_pending();
  }
  if (is_act16(x, dimX[0], dimX[1], dimX[2], dimX[3])) {
    launch_add_act_bf16(act16_ptr(x), nullptr, nullptr, (int)dimX[1], (bf16 *)y, n, act, 0.f,
                        0.f, mode_f16(), r.stream);
    mark_act16(y, dimX[0], dimX[1], dimX[2], dimX[3]);
    return y;
  }
  ensure_f32(x);
  launch_act_f32(x, y, n, act, 0.f, 0.f, r.stream);
  mark_f32(y);
  return y;
}

float *CUDAClipFunc(float *x, float *y, int64_t *dimOut, float lo, float hi, int64_t rank) {
  Runtime &r = rt();
  const int64_t n = prod(dimOut, rank);
  CallScope scope;
  Entry e = trace_entry(S_CLIP);
  int at = 0;
  put(e, {x, y});
  put(e, at, rank); put(e, at, dimOut, rank);
  e.args.f[0] = lo; e.args.f[1] = hi;
  te_ptr(e, x); te_ptr(e, y); te_dims(e, dimOut, (int)rank); te_f(e, lo); te_f(e, hi);
  e.in[0] = (uintptr_t)x; e.in_bytes[0] = n * 4; e.out = (uintptr_t)y; e.out_bytes = n * 4;
  for (int i = 0; i < 4 && i < rank; ++i) e.dims[i] = dimOut[i];
  e.kind = rank == 4 ? CK_CLIP : CK_NONE;
  const Role role = step(e, false);
  if (role == R_SKIP) return y;
  if (role == R_ABSORB && g_pending.active) {
    const ConvGeom &g = g_pending.g;
    if (rank == 4 && x == g_pending.out && !g_pending.act_set && dimOut[0] == g.N &&
        dimOut[1] == g.K && dimOut[2] == g.P && dimOut[3] == g.Q) {
      pending_retarget(y);
      g_pending.g.act = ACT_CLIP;
      g_pending.g.lo = lo;
      g_pending.g.hi = hi;
      g_pending.act_set = true;
      if (!g_pending.linked) flush_pending();
      return y;
    }
    flush_pending();
  }
  if (rank == 4 && is_act16(x, dimOut[0], dimOut[1], dimOut[2], dimOut[3])) {
    launch_add_act_bf16(act16_ptr(x), nullptr, nullptr, (int)dimOut[1], (bf16 *)y, n, ACT_CLIP,
                        lo, hi, mode_f16(), r.stream);
    mark_act16(y, dimOut[0], dimOut[1], dimOut[2], dimOut[3]);
    return y;
  }
  ensure_f32(x);
  launch_act_f32(x, y, n, ACT_CLIP, lo, hi, r.stream);
  mark_f32(y);
  return y;
}

float *DNNTensorOpFunc(cudnnContext *, int64_t opMode, float *A, int64_t *dimA, int32_t rankA,
                       float *B, int64_t *dimB, int32_t rankB, float *out, int64_t *dimOut,
                       int32_t rankOut, float bias) {
  Runtime &r = rt();
  (void)dimOut;
  (void)rankOut;
  const bool rank_ok = rankA <= 8 && rankB <= rankA && rankA >= 1;
  // B's shape padded with leading 1s to A's rank
  int64_t dB[8] = {1, 1, 1, 1, 1, 1, 1, 1};
  if (rank_ok)
    for (int i = 0; i < rankA; ++i) dB[i] = i < rankA - rankB ? 1 : dimB[i - (rankA - rankB)];
  bool same = rank_ok && rankA == 4;
  for (int i = 0; same && i < 4; ++i) same = dB[i] == dimA[i];
  const bool bias_shape = rank_ok && rankA == 4 && dB[0] == 1 && dB[1] == dimA[1] && dB[2] == 1 &&
                          dB[3] == 1 && !same;

  CallScope scope;
  Entry e = trace_entry(S_TENSOR_OP);
  int at = 0;
  put(e, {A, B, out});
  put(e, at, opMode); put(e, at, rankA); put(e, at, rankB);
  if (rank_ok) { put(e, at, dimA, rankA); put(e, at, dimB, rankB); }
  e.args.f[0] = bias;
  te_ptr(e, A); te_ptr(e, B); te_ptr(e, out);
  te_i(e, opMode); te_f(e, bias);
  if (rank_ok) { te_dims(e, dimA, rankA); te_dims(e, dB, rankA); }
  e.in[0] = (uintptr_t)A; e.in[1] = opMode == 4 ? 0 : (uintptr_t)B; e.out = (uintptr_t)out;
  e.out_bytes = rank_ok ? prod(dimA, rankA) * 4 : 0;
  e.in_bytes[0] = e.out_bytes;
  e.in_bytes[1] = rank_ok ? prod(dB, rankA) * 4 : 0;
  for (int i = 0; i < 4 && i < rankA; ++i) e.dims[i] = dimA[i];
  if (opMode == 0 && bias == 1.0f) e.kind = bias_shape ? CK_BIAS_ADD : (same ? CK_SAME_ADD : CK_NONE);
  if (opMode == 0 && bias == 1.0f && rank_ok && rankA == 2 && dB[0] == 1 && dB[1] == dimA[1]) e.kind = CK_ROW_BIAS;
  const Role role = step(e, false);
  if (role == R_SKIP) return out;

  if (!rank_ok) {
    set_error(996, "tensor op: unsupported rank");
    return out;
  }
  if (role == R_ABSORB && g_pending.active) {
    const ConvGeom &g = g_pending.g;
    const bool dims_ok = dimA[0] == g.N && dimA[1] == g.K &&
                         (rankA == 2 ? g_pending.product : dimA[2] == g.P && dimA[3] == g.Q);
    if ((e.kind == CK_BIAS_ADD || e.kind == CK_ROW_BIAS) && dims_ok && A == g_pending.out && !g_pending.bias_set &&
        !g_pending.res_set && !g_pending.act_set) {
      const float *bd = resident_f32(B, (size_t)g.K * 4);
      bool ready = g_pack_was_resident;
      const void *block_b = nullptr;
      if (g_pending.linked && (!g_pending.depthwise || mode_f16())) {
        block_b = g_pending.depthwise ? packed_for_block(B, PACK_IR_HALF, (size_t)g.K * 2, g.K, 1)
                                      : packed_for_block(B, PACK_BIAS3, (size_t)g.K * 32, g.K, 0);
        ready = ready && g_pack_was_resident;
      }
      if (g_pending.active) {   // (an upload of B may have had to run it early)
        if (g_pending.depthwise) g_pending.bias = bd;
        else g_pending.a.bias = bd;
        g_pending.block_b = block_b;
        job_track_bias(g_pending, bd, B, g.K);
        if (!ready) g_pending.a.consts_ready = 0;
        g_pending.bias_set = true;
        pending_retarget(out);
        return out;
      }
    }
    if (g_pending.active && e.kind == CK_SAME_ADD && dims_ok && !g_pending.depthwise && !g_pending.product && !g_pending.res_set &&
        !g_pending.act_set && ((A == g_pending.out) != (B == g_pending.out))) {
      const float *other = A == g_pending.out ? B : A;
      if (g_pending.after_summand && other == g_front[0].out && join_summands(g_front[0], g_pending)) {
        if (g_front[0].absorbed) trace_count_chain();
        g_pending.after_summand = false;
        g_fronts = 0;
        g_pending.res_set = true;
        if (other != out) elide(const_cast<float *>(other));
        pending_retarget(out);
        return out;
      }
      launch_summand();
      const bool parts = g_pending.a.split && g.K % 16 == 0 && is_parts(other, g.N, g.K, g.P, g.Q);
      if (parts || (!g_pending.a.split && is_act16(other, g.N, g.K, g.P, g.Q))) {
        g_pending.a.residual = act16_ptr(other);
        g_pending.res_set = true;
        if ((const void *)g_pending.a.residual == other) {
          g_pending.dep_lo[1] = (uintptr_t)other;
          g_pending.dep_hi[1] = (uintptr_t)other + (size_t)g.N * g.K * g.P * g.Q * 2;
        }
        pending_retarget(out);
        return out;
      }
    }
    flush_pending();
  }
  if (opMode == 0 && rankA == 4 && bias == 1.0f &&
      is_act16(A, dimA[0], dimA[1], dimA[2], dimA[3])) {
    const int64_t n = numel4(dimA);
    if (same && is_act16(B, dimA[0], dimA[1], dimA[2], dimA[3])) {
      launch_add_act_bf16(act16_ptr(A), act16_ptr(B), nullptr, (int)dimA[1], (bf16 *)out, n,
                          ACT_IDENTITY, 0.f, 0.f, mode_f16(), r.stream);
      mark_act16(out, dimA[0], dimA[1], dimA[2], dimA[3]);
      return out;
    }
    if (bias_shape) {
      // a bias vector uploaded from host memory is kept resident like the filters are
      const float *bd = resident_f32(B, (size_t)dimA[1] * 4);
      launch_add_act_bf16(act16_ptr(A), nullptr, bd, (int)dimA[1], (bf16 *)out, n, ACT_IDENTITY,
                          0.f, 0.f, mode_f16(), r.stream);
      mark_act16(out, dimA[0], dimA[1], dimA[2], dimA[3]);
      return out;
    }
  }
  ensure_f32(A);
  // a small constant (the C operand of a Gemm, say) is read from its resident copy
  const float *Bd = opMode != 4 ? operand_f32(B, (size_t)prod(dB, rankA) * 4) : B;
  if (opMode != 0 && opMode != 1 && opMode != 4) {
    set_error(996, "tensor op: unsupported mode");
    return out;
  }
  launch_tensor_op_f32((int)opMode, A, Bd, out, rankA, dimA, dB, bias, r.stream);
  mark_f32(out);
  return out;
}

// ---------------------------------------------------------------- pooling / reduction
static float *pool_common(int sym, float *x, int64_t *dI, float *y, int64_t *dO, int64_t *kernel,
                          int64_t *padding, int64_t *stride, bool avg) {
  Runtime &r = rt();
  const int N = (int)dI[0], C = (int)dI[1], H = (int)dI[2], W = (int)dI[3];
  const int P = (int)dO[2], Q = (int)dO[3];
  const int ph = (int)padding[0], pw = (int)padding[2];
  CallScope scope;
  Entry e = trace_entry(sym);
  int at = 0;
  put(e, {x, y});
  put(e, at, dI, 4); put(e, at, dO, 4); put(e, at, kernel, 2); put(e, at, padding, 4); put(e, at, stride, 2);
  te_ptr(e, x); te_ptr(e, y); te_dims(e, dI, 4); te_dims(e, dO, 4); te_dims(e, kernel, 2);
  te_dims(e, padding, 4); te_dims(e, stride, 2);
  e.in[0] = (uintptr_t)x; e.in_bytes[0] = numel4(dI) * 4; e.out = (uintptr_t)y;
  e.out_bytes = numel4(dO) * 4;
  if (!avg && kernel[0] == 3 && kernel[1] == 3 && stride[0] == 2 && stride[1] == 2 && ph == 1 &&
      pw == 1 && padding[1] == 1 && padding[3] == 1)
    e.kind = CK_POOL_3S2;
  if (!avg && kernel[0] == 2 && kernel[1] == 2 && stride[0] == 2 && stride[1] == 2 && !padding[0] && !padding[1] &&
      !padding[2] && !padding[3] && P == H / 2 && Q == W / 2)
    e.kind = CK_POOL_2S2;
  const Role role = step(e, false);
  if (role == R_SKIP) return y;
  const bool for_matmul = (trace_last_flags() & RF_FOR_MATMUL) != 0;
  if (role == R_ABSORB && g_pending.active) {
    // the held-back stem convolution and this pool run as one kernel
    ConvJob &j = g_pending;
    const ConvGeom &g = j.g;
    bool done = false;
    if (!j.depthwise && j.w_stem && !j.res_set && x == j.out && N == g.N && C == g.K && H == g.P &&
        W == g.Q && e.kind == CK_POOL_3S2) {
      StemPoolArgs sa;
      memset(&sa, 0, sizeof(sa));
      sa.x = j.a.x;
      sa.bias = j.a.bias;
      sa.y = (bf16 *)y;
      sa.N = g.N; sa.H = g.H; sa.row_bytes = j.a.row_elems * 2; sa.w_step_bytes = j.a.w_step * 2;
      sa.P = g.P; sa.Q = g.Q; sa.K = g.K; sa.R = g.R; sa.Cf = j.a.Cf;
      sa.pad_h = g.pad_h; sa.stride_h = g.stride_h;
      sa.PP = P; sa.QP = Q;
      sa.lo = j.a.act == ACT_RELU ? 0.0f : (j.a.act == ACT_CLIP ? j.a.lo : -INFINITY);
      sa.hi = j.a.act == ACT_CLIP ? j.a.hi : INFINITY;
      sa.w = j.w_stem;
      sa.w_fold = j.a.w;
      if (stem_pool_supported(sa)) {
        if (launch_stem_pool(sa, r.dev_err, r.num_sms, r.stream)) {
          j.active = false;
          j.absorbed++;
          elide(j.out);
          trace_count_chain();
          mark_act16(y, N, C, P, Q);
          done = true;
        }
      }
    }
    if (done) return y;
    if (e.kind == CK_POOL_2S2 && !for_matmul && !j.depthwise && !j.product && !j.linked && !j.joined && !j.res_set && !j.a.split &&
        j.a.Cf == g.C && x == j.out && N == g.N && C == g.K && H == g.P && W == g.Q) {
      TcConvArgs a = j.a;
      a.act = g.act; a.lo = g.lo; a.hi = g.hi;
      a.y = (bf16 *)16;
      a.bias = nullptr;
      a.consts_ready = 0;
      if (tc_conv_takes_pool(a)) {
        elide(j.out);
        j.out = y;
        j.g.P = P;
        j.g.Q = Q;
        j.a.pool2 = 1;
        j.absorbed++;
        flush_pending();
        return y;
      }
    }
    flush_pending();
  }
  if (r.mode != MATH_FP32 && C % 8 == 0 && is_act16(x, N, C, H, W)) {
    // read by a Flatten and the product behind it: where the Flatten need not move it
    void *home = for_matmul ? home_acquire((size_t)N * C * P * Q * 2) : nullptr;
    launch_pool_bf16(act16_ptr(x), (bf16 *)(home ? home : y), N, C, H, W, P, Q, (int)kernel[0], (int)kernel[1],
                     ph, pw, (int)stride[0], (int)stride[1], avg, mode_f16(), r.stream);
    mark_act16(y, N, C, P, Q, home);
    return y;
  }
  if (r.mode == MATH_FP32 && is_parts(x, N, C, H, W)) {
    void *home = home_acquire((size_t)N * C * P * Q * 6);
    if (home) {
      launch_pool3(act16_ptr(x), (bf16 *)home, N, C, H, W, P, Q, (int)kernel[0], (int)kernel[1], ph, pw,
                   (int)stride[0], (int)stride[1], avg, r.stream);
      mark_parts(y, N, C, P, Q, home);
      return y;
    }
  }
  ensure_f32(x);
  launch_pool_f32(x, y, N, C, H, W, P, Q, (int)kernel[0], (int)kernel[1], ph, pw, (int)stride[0],
                  (int)stride[1], avg, r.stream);
  mark_f32(y);
  return y;
}

float *DNNMaxPoolFunc(cudnnContext *, float *x, int64_t dimIn[4], float *y, int64_t dimOut[4],
                      int64_t kernel[2], int64_t padding[4], int64_t stride[2]) {
  return pool_common(S_MAXPOOL, x, dimIn, y, dimOut, kernel, padding, stride, false);
}

float *DNNAveragePoolFunc(cudnnContext *, float *x, int64_t dimIn[4], float *y, int64_t dimOut[4],
                          int64_t kernel[2], int64_t padding[4], int64_t stride[2]) {
  return pool_common(S_AVGPOOL, x, dimIn, y, dimOut, kernel, padding, stride, true);
}

float *DNNReduceFunc(cudnnContext *, int32_t rank, float *x, int64_t *dimIn, float *y,
                     int64_t *dimOut, int32_t mode) {
  Runtime &r = rt();
  CallScope scope;
  Entry e = trace_entry(S_REDUCE);
  int at = 0;
  put(e, {x, y});
  put(e, at, rank); put(e, at, mode);
  if (rank <= 8 && rank > 0) { put(e, at, dimIn, rank); put(e, at, dimOut, rank); }
  te_ptr(e, x); te_ptr(e, y); te_i(e, mode);
  if (rank <= 8 && rank > 0) { te_dims(e, dimIn, rank); te_dims(e, dimOut, rank); }
  e.in[0] = (uintptr_t)x; e.out = (uintptr_t)y;
  e.out_bytes = rank <= 8 && rank > 0 ? prod(dimOut, rank) * 4 : 0;
  e.in_bytes[0] = rank <= 8 && rank > 0 ? prod(dimIn, rank) * 4 : 0;
  if (step(e, false) == R_SKIP) return y;
  const bool for_matmul = (trace_last_flags() & RF_FOR_MATMUL) != 0;
  if (mode != 5 || rank > 8) {
    set_error(995, "reduce: only mode 5 (mean) is implemented");
    return y;
  }
  if (rank == 4 && dimOut[2] == 1 && dimOut[3] == 1 && dimOut[0] == dimIn[0] &&
      dimOut[1] == dimIn[1] && dimIn[1] % 8 == 0 &&
      is_act16(x, dimIn[0], dimIn[1], dimIn[2], dimIn[3])) {
    void *home = for_matmul ? home_acquire((size_t)(dimIn[0] * dimIn[1]) * 2) : nullptr;
    launch_gap_bf16(act16_ptr(x), y, (bf16 *)home, (int)dimIn[0], (int)(dimIn[2] * dimIn[3]), (int)dimIn[1],
                    mode_f16(), r.stream);
    if (home) mark_act16(y, dimIn[0], dimIn[1], 1, 1, home);
    else mark_f32(y);
    return y;
  }
  if (r.mode == MATH_FP32 && rank == 4 && dimOut[2] == 1 && dimOut[3] == 1 && dimOut[0] == dimIn[0] &&
      dimOut[1] == dimIn[1] && is_parts(x, dimIn[0], dimIn[1], dimIn[2], dimIn[3])) {
    launch_gap3(act16_ptr(x), y, (int)dimIn[0], (int)(dimIn[2] * dimIn[3]), (int)dimIn[1], r.stream);
    mark_f32(y);
    return y;
  }
  ensure_f32(x);
  launch_reduce_mean_f32(x, y, rank, dimIn, dimOut, r.stream);
  mark_f32(y);
  return y;
}

// ---------------------------------------------------------------- classifier head
float *CUBLASMatmul2dFunc(int64_t /*rank*/, float *A, int64_t dimA[2], float *B, int64_t dimB[2],
                          float * /*C*/, int64_t * /*dimC*/, float *out, int64_t * /*dimOut*/,
                          float alpha, float beta, int64_t transA, int64_t transB) {
  Runtime &r = rt();
  const int M = (int)(transA ? dimA[1] : dimA[0]);
  const int K = (int)(transA ? dimA[0] : dimA[1]);
  const int N = (int)(transB ? dimB[0] : dimB[1]);
  CallScope scope;
  Entry e = trace_entry(S_MATMUL);
  int at = 0;
  put(e, {A, B, out});
  put(e, at, dimA, 2); put(e, at, dimB, 2); put(e, at, transA); put(e, at, transB);
  e.args.f[0] = alpha; e.args.f[1] = beta;
  te_ptr(e, A); te_ptr(e, B); te_ptr(e, out); te_dims(e, dimA, 2); te_dims(e, dimB, 2);
  te_f(e, alpha); te_f(e, beta); te_i(e, transA); te_i(e, transB);
  e.in[0] = (uintptr_t)A; e.in[1] = (uintptr_t)B; e.in[2] = beta != 0.0f ? (uintptr_t)out : 0;
  e.out = (uintptr_t)out; e.out_bytes = (int64_t)M * N * 4;
  e.in_bytes[0] = dimA[0] * dimA[1] * 4; e.in_bytes[1] = dimB[0] * dimB[1] * 4;
  e.in_bytes[2] = e.out_bytes;
  e.dims[0] = M; e.dims[1] = N;
  const bool out_zero = is_zero(out);
  const bool parts = r.mode == MATH_FP32;
  e.fusable = !transA && transB && alpha == 1.0f && (beta == 0.0f || out_zero) && M > 0 &&
              (parts ? fp32_on_tensor_cores() && (double)form_images(M) * N * K >= 1e6 : K % 16 == 0);
  const Role role = step(e, false);
  if (role == R_SKIP) return out;
  if (r.log) fprintf(stderr, "[occamy] matmul2d M%d N%d K%d tA%d tB%d\n", M, N, K, (int)transA, (int)transB);
  if (e.fusable) {
    ConvJob job;
    TcConvArgs &a = job.a;
    memset(&a, 0, sizeof(a));
    const int Kp = (K + 15) / 16 * 16;
    a.split = parts ? 1 : 0;
    a.N = 1; a.H = 1; a.W = M; a.Cf = Kp; a.K = N; a.P = 1; a.Q = M; a.R = 1; a.S = 1;
    a.stride_h = a.stride_w = 1;
    a.form_n = form_n(M);
    a.act = ACT_IDENTITY;
    a.f16 = mode_f16() ? 1 : 0;
    int c = K;   // channels of A where it is an image that a Flatten passed on
    uintptr_t base = 0;
    const TensorRec *rec = reg_find(A, &base);
    const bool image = !parts && rec && base == (uintptr_t)A && is_act16(A, rec->n, rec->c, rec->h, rec->w) && rec->n == M &&
                       rec->c * rec->h * rec->w == K && rec->h * rec->w <= 64 && rec->c % 16 == 0;
    if (image && rec->h * rec->w > 1) {
      // NHWC rows against [N][c][h][w] filters: a convolution whose filter covers the whole image
      c = (int)rec->c;
      a.N = M; a.H = (int)rec->h; a.W = (int)rec->w; a.Cf = c; a.P = a.Q = 1; a.R = a.H; a.S = a.W;
    }
    a.out_f32 = out;
    a.out_nchw = a.R * a.S > 1;
    a.ldo = N;
    a.x = (const bf16 *)16;
    a.w = (const bf16 *)16;
    if (tc_conv_supported(a)) {
      if (image) {
        a.x = act16_ptr(A);
        if ((const void *)a.x == A) {
          job.dep_lo[0] = (uintptr_t)A;
          job.dep_hi[0] = (uintptr_t)A + (size_t)M * K * 2;
        }
      } else if (parts) {
        ensure_f32(A);
        bf16 *as = (bf16 *)scratch_get(0, (size_t)6 * M * Kp);
        if (as) launch_split3_rows(A, as, M, K, Kp, (int)dimA[1], r.stream);
        a.x = as;
      } else {
        ensure_f32(A);
        bf16 *ab = (bf16 *)scratch_get(0, (size_t)M * K * 2);
        launch_f32_to_bf16(A, ab, (int64_t)M * K, mode_f16(), r.stream);
        a.x = ab;
      }
      a.w = (const bf16 *)(parts ? packed_weights(B, PACK_PARTS, (size_t)6 * N * Kp, N, K, 1, 1, 0, Kp)
                                 : packed_weights(B, PACK_KRSC, (size_t)N * K * 2, N, c, a.R, a.S, 0, c));
      if (a.x && a.w) {
        a.consts_ready = g_pack_was_resident ? 1 : 0;
        a.out_f32 = nullptr;
        a.out_nchw = 0;
        ConvGeom &g = job.g;
        memset(&g, 0, sizeof(g));
        g.N = M; g.K = N; g.P = g.Q = 1; g.C = c; g.H = a.H; g.W = a.W; g.R = a.R; g.S = a.S;
        g.groups = g.stride_h = g.stride_w = 1;
        g.act = ACT_IDENTITY;
        job.product = true;
        job.out16 = !parts && (trace_last_flags() & RF_FOR_MATMUL) && N % 16 == 0;
        job.out = out;
        if (role == R_DEFER) {
          g_pending = job;
          g_pending.active = true;
          return out;
        }
        launch_job(job);
        return out;
      }
    }
  }
  ensure_f32(A);
  const float *Bd = operand_f32(B, (size_t)(dimB[0] * dimB[1]) * 4);
  if (beta != 0.0f) ensure_f32(out);
  launch_gemm_f32(A, Bd, out, M, N, K, (int)dimA[1], (int)dimB[1], alpha, out_zero ? 0.0f : beta,
                  transA != 0, transB != 0, r.stream);
  mark_f32(out);
  return out;
}

float *CUDASoftmaxFunc(float *x, int64_t *dimIn, float *y, int64_t * /*dimOut*/, int64_t axis,
                       int64_t rank) {
  Runtime &r = rt();
  if (axis < 0) axis += rank;
  int64_t outer = 1, inner = 1;
  for (int64_t i = 0; i < axis; ++i) outer *= dimIn[i];
  for (int64_t i = axis + 1; i < rank; ++i) inner *= dimIn[i];
  CallScope scope;
  Entry e = trace_entry(S_SOFTMAX);
  int at = 0;
  put(e, {x, y});
  put(e, at, axis); put(e, at, rank); put(e, at, dimIn, rank);
  te_ptr(e, x); te_ptr(e, y); te_dims(e, dimIn, (int)rank); te_i(e, axis);
  e.in[0] = (uintptr_t)x; e.out = (uintptr_t)y; e.out_bytes = prod(dimIn, rank) * 4;
  e.in_bytes[0] = e.out_bytes;
  if (step(e, false) == R_SKIP) return y;
  ensure_f32(x);
  launch_softmax_f32(x, y, outer, dimIn[axis], inner, r.stream);
  mark_f32(y);
  return y;
}

static float *copy_common(int sym, float *x, int64_t *dimIn, int64_t rank, float *y) {
  Runtime &r = rt();
  const int64_t n = prod(dimIn, rank);
  CallScope scope;
  Entry e = trace_entry(sym);
  int at = 0;
  put(e, {x, y});
  put(e, at, rank); put(e, at, dimIn, rank);
  te_ptr(e, x); te_ptr(e, y); te_dims(e, dimIn, (int)rank);
  e.in[0] = (uintptr_t)x; e.in_bytes[0] = n * 4; e.out = (uintptr_t)y; e.out_bytes = n * 4;
  if (step(e, false) == R_SKIP) return y;
  // A tensor in a buffer of its own goes by its record: the same values in the same logical order.
  if (sym == S_FLATTEN && rank == 4 && is_act16(x, dimIn[0], dimIn[1], dimIn[2], dimIn[3]) &&
      (const void *)act16_ptr(x) != x) {
    pending_guard_range(y, (size_t)n * 4, true);
    mark_act16(y, dimIn[0], dimIn[1], dimIn[2], dimIn[3], act16_ptr(x));
    return y;
  }
  ensure_f32(x);
  enqueue_copy(y, x, (size_t)n * 4, r.stream);
  mark_f32(y);
  return y;
}

float *CUDAFlattenFunc(float *x, int64_t *dimIn, float *y, int64_t * /*dimOut*/, int32_t /*axis*/,
                       int64_t rank) {
  return copy_common(S_FLATTEN, x, dimIn, rank, y);
}

float *CUDAReshapeFunc(float *x, int64_t *dimIn, int64_t rank, float *y) {
  return copy_common(S_RESHAPE, x, dimIn, rank, y);
}

// Called by the entry points outside this file: they take part in no chain and their
// reads are not tracked, so they end the speculation for this inference.
void occamy_internal_opaque_call(void) {
  graph_settle();
  Entry e = trace_entry(S_OPAQUE);
  step(e, false);
  settle_sources();
}

}  // extern "C"

// Whether the convolution of entry `e` reads its input in the 16-bit path's form, whatever the mode it was
// recorded in: wider than that, Entry::fusable goes by channel counts alone.
bool occ::entry_reads_16(const Entry &e) {
  const int64_t *v = e.args.v;   // dX[4], dW[4], pads[2], strides[2], groups, activation mode
  ConvGeom g;
  float lo, hi;
  const int act = act_of_mode(v[13], lo, hi);
  if (!conv_geometry(v, v + 4, v[12], v + 8, v + 10, act, lo, hi, g) || g.P <= 0 || g.Q <= 0 || g.N <= 0) return false;
  if (g.groups > 1) return g.groups == g.C && g.K == g.C && g.C % 8 == 0;   // as prepare_depthwise()
  TcConvArgs a;
  int Cp, Sp, Wp;
  return dense_args(g, a, Cp, Sp, Wp);
}

// Whether the convolution of entry `e` takes a 2x2 max pool behind it along.
bool occ::entry_takes_pool(const Entry &e) {
  const int64_t *v = e.args.v;   // dX[4], dW[4], pads[2], strides[2], groups
  if (!e.fusable || e.parts || e.depthwise || v[1] % 16 || v[12] != 1) return false;
  TcConvArgs a;
  memset(&a, 0, sizeof(a));
  a.N = (int)v[0]; a.H = (int)v[2]; a.W = (int)v[3]; a.Cf = (int)v[1];
  a.K = (int)v[4]; a.R = (int)v[6]; a.S = (int)v[7];
  a.P = (int)e.dims[2]; a.Q = (int)e.dims[3];
  a.pad_h = (int)v[8]; a.pad_w = (int)v[9]; a.stride_h = (int)v[10]; a.stride_w = (int)v[11];
  a.act = ACT_RELU;
  a.f16 = mode_f16() ? 1 : 0;
  a.x = a.w = (const bf16 *)16;
  a.y = (bf16 *)16;
  return tc_conv_takes_pool(a);
}

// ---------------------------------------------------------------- made again
void occ::flush_held_back() { flush_pending(); }
bool occ::anything_held_back() { return g_pending.active; }

// The call of entry `e`, its pointers where `place` says; `host` is the source of a constant.
void occ::run_again(const Entry &e, const std::function<void *(void *)> &place, const void *host) {
  void *p[4];
  for (int k = 0; k < 4; ++k) p[k] = place(e.args.p[k]);
  float *const f[4] = {(float *)p[0], (float *)p[1], (float *)p[2], (float *)p[3]};
  int64_t v[24];
  memcpy(v, e.args.v, sizeof(v));
  switch (e.sym) {
    case S_MEMOFFSET: hand_out(p[0], (size_t)v[0]); break;
    case S_H2D: wrapDNNMemcpy(p[0], host, (size_t)v[0], 1, nullptr); break;
    case S_CONV:
      DNNConvFunc(nullptr, f[0], v, f[1], v + 4, nullptr, 0, 0, v[12], v + 8, v + 10, f[3]);
      break;
    case S_CONV_BIAS_ACT:
      DNNConvBiasActivFunc(nullptr, f[0], v, f[1], v + 4, f[2], v, nullptr, 0, 0, v + 8, v + 10, v[13], f[3]);
      break;
    case S_ACTIVE: DNNActiveFunc(nullptr, f[0], v, (int32_t)v[4], f[1]); break;
    case S_CLIP: CUDAClipFunc(f[0], f[1], v + 1, e.args.f[0], e.args.f[1], v[0]); break;
    case S_TENSOR_OP:
      DNNTensorOpFunc(nullptr, v[0], f[0], v + 3, (int32_t)v[1], f[1], v + 3 + v[1], (int32_t)v[2], f[2], v + 3,
                      (int32_t)v[1], e.args.f[0]);
      break;
    case S_MAXPOOL: DNNMaxPoolFunc(nullptr, f[0], v, f[1], v + 4, v + 8, v + 10, v + 14); break;
    case S_AVGPOOL: DNNAveragePoolFunc(nullptr, f[0], v, f[1], v + 4, v + 8, v + 10, v + 14); break;
    case S_REDUCE: DNNReduceFunc(nullptr, (int32_t)v[0], f[0], v + 2, f[1], v + 2 + v[0], (int32_t)v[1]); break;
    case S_MATMUL:
      CUBLASMatmul2dFunc(2, f[0], v, f[1], v + 2, f[2], v, f[2], v, e.args.f[0], e.args.f[1], v[4], v[5]);
      break;
    case S_SOFTMAX: CUDASoftmaxFunc(f[0], v + 2, f[1], v + 2, v[0], v[1]); break;
    case S_FLATTEN: CUDAFlattenFunc(f[0], v + 1, f[1], v + 1, 1, v[0]); break;
    case S_RESHAPE: CUDAReshapeFunc(f[0], v + 1, v[0], f[1]); break;
    default: break;   // a window holds no other calls
  }
}

extern "C" {
// ---------------------------------------------------------------- controls
void occamy_set_math_mode(int mode) {
  graph_settle();
  flush_pending();   // what is held back was prepared for the mode it arrived in
  rt().mode = mode == 0 ? MATH_FP32 : (mode == 2 ? MATH_F16 : MATH_BF16);
}
int occamy_get_math_mode(void) { return (int)rt().mode; }

int occamy_last_error(int clear) {
  Runtime &r = rt();
  if (r.last_error == 0) {   // a watchdog report of the allocation-free entry point, if any
    const int na = noalloc_poll_error(clear != 0);
    if (na > 0) set_error(na, "kernel watchdog (occamy_conv_bias_act_noalloc)");
  }
  const int e = r.last_error;
  if (clear) r.last_error = 0;
  return e;
}

int occamy_synchronize(void) {
  Runtime &r = rt();
  graph_settle();
  flush_pending();
  settle_sources();
  cudaError_t e = cudaStreamSynchronize(r.stream);
  if (e != cudaSuccess) set_error((int)e, "synchronize");
  poll_watchdog();
  const int na = noalloc_poll_error(true);
  if (na > 0) set_error(na, "kernel watchdog (occamy_conv_bias_act_noalloc)");
  return (int)e;
}

cudaStream_t occamy_stream(void) {
  rt();
  graph_settle();   // the caller may order work of its own behind the calls made so far
  flush_pending();
  settle_sources();
  return rt().stream;
}

void occamy_selftest_bounded_wait(void) {
  graph_settle();
  flush_pending();
  launch_selftest_bounded_wait(rt().stream);
}

void occamy_get_counters(int64_t out[8]) {
  Runtime &r = rt();
  for (int i = 0; i < 8; ++i) out[i] = r.counters[i];
}

int occamy_get_form_counters(int64_t *out, int n) {
  constexpr int FORMS = CNT_COUNT - CNT_SPLIT_REDUCTION;
  for (int i = 0; i < n && i < FORMS; ++i) out[i] = rt().counters[CNT_SPLIT_REDUCTION + i];
  return FORMS;
}

int64_t occamy_fused_chains(void) { return trace_fused_chains(); }
void occamy_clear_weight_cache(void);

void occamy_profile_begin(void) {
  Runtime &r = rt();
  graph_settle();
  r.prof_count = 0;
  r.profiling = true;
}

int occamy_profile_end(float *ms, int cap) {
  Runtime &r = rt();
  graph_settle();
  flush_pending();
  r.profiling = false;
  OCC_CUDA(cudaStreamSynchronize(r.stream));
  const int n = r.prof_count;
  for (int i = 0; i < n && i < cap; ++i) {
    float t = 0.f;
    OCC_CUDA(cudaEventElapsedTime(&t, r.prof_events[2 * i], r.prof_events[2 * i + 1]));
    ms[i] = t;
  }
  r.prof_count = 0;
  return n;
}

void occamy_set_cross_call_fusion(int on) {
  graph_settle();
  flush_pending();
  trace_set_enabled(on != 0);
}

void occamy_set_fp32_tensor_cores(int on) {
  graph_settle();
  g_fp32_tc = on ? 1 : 0;
}

void occamy_set_weight_cache(int on) {
  graph_settle();
  if (!on) occamy_clear_weight_cache();
  rt().cache_weights = on != 0;
}

void occamy_clear_weight_cache(void) {
  Runtime &r = rt();
  graph_settle();
  graph_forget_all();
  flush_pending();
  OCC_CUDA(cudaStreamSynchronize(r.stream));
  for (auto &kv : r.wcache)
    if (kv.second.dev) cudaFree(kv.second.dev);
  r.wcache.clear();
  r.resident.clear();
  graph_free_memory();
  free_idle_homes();
}

}  // extern "C"
