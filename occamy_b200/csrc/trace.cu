// Recording, matching and analysis of per-inference call traces (see trace.h).
#include "trace.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "kernels.h"
#include "runtime.h"

namespace occ {

namespace {

struct TraceState {
  int enabled = -1;
  bool in_inference = false;
  bool matched_so_far = false;   // at least one recorded program still matches
  std::vector<Entry> rec;        // calls of this inference behind the adopted prefix
  TraceProgram *prefix = nullptr;   // program whose first prefix_len calls this inference made in one go
  size_t prefix_len = 0;
  std::vector<TraceProgram> programs;
  std::vector<int> cands;
  uintptr_t pool_base = 0;
  size_t pool_bytes = 0;
  uintptr_t last_pool_base = 0;   // the pool of this inference, also after it was given back
  size_t last_pool_bytes = 0;
  uint16_t last_flags = 0;
  int forced = -1;               // role of the next call, see trace_force()
  int elided = 0;
  int64_t fused_chains = 0;
};

// never destroyed: recorded programs own CUDA graphs, and the driver may be gone by then
TraceState &g_ts = *new TraceState;

constexpr size_t MAX_ENTRIES = 50000;
constexpr size_t MAX_PROGRAMS = 16;

// One multiply per value: an entry has about twenty of them and a ResNet-50 inference 330 entries.
inline void mix(uint64_t &h, uint64_t v) {
  h = (h ^ v) * 0x9e3779b97f4a7c15ull;
  h ^= h >> 32;
}

bool overlaps(uintptr_t a, int64_t abytes, uintptr_t b, int64_t bbytes) {
  return a < b + (uintptr_t)bbytes && b < a + (uintptr_t)abytes;
}

bool is_passive(int sym) {
  return sym == S_MEMOFFSET || sym == S_MALLOC || sym == S_H2D || sym == S_DEALLOC;
}

// True when nothing reads [p, p+bytes) from entry `from` on until the range is handed out
// again, freed, or the inference ends.
bool dies_unread(const std::vector<Entry> &rec, uintptr_t p, int64_t bytes, size_t from) {
  for (size_t t = from; t < rec.size(); ++t) {
    const Entry &e = rec[t];
    for (int k = 0; k < 3; ++k)   // any overlap with an input counts as a read
      if (e.in[k] && overlaps(e.in[k], e.in_bytes[k] > 0 ? e.in_bytes[k] : 1, p, bytes)) return false;
    if ((e.sym == S_MEMOFFSET || e.sym == S_MALLOC) && overlaps(e.out, e.out_bytes, p, bytes))
      return true;
    if ((e.sym == S_DEALLOC && e.out == p) || e.sym == S_POOLFREE) return true;
    if (e.sym == S_OPAQUE) return false;
  }
  return true;
}

bool same_dims(const Entry &a, const Entry &b) {
  return a.dims[0] == b.dims[0] && a.dims[1] == b.dims[1] && a.dims[2] == b.dims[2] &&
         a.dims[3] == b.dims[3];
}

// True when what reads [p, p+bytes) from entry `from` on, until the range is handed out again or
// freed, are matrix products (as their first operand) and Flattens whose result only such read.
bool only_matmuls_read(const std::vector<Entry> &rec, uintptr_t p, int64_t bytes, size_t from) {
  bool any = false;
  for (size_t t = from; t < rec.size(); ++t) {
    const Entry &e = rec[t];
    for (int k = 0; k < 3; ++k) {
      if (!e.in[k] || !overlaps(e.in[k], e.in_bytes[k] > 0 ? e.in_bytes[k] : 1, p, bytes)) continue;
      const bool product = e.sym == S_MATMUL && k == 0 && e.in[0] == p && e.fusable;
      const bool flat = e.sym == S_FLATTEN && e.in[0] == p && only_matmuls_read(rec, e.out, e.out_bytes, t + 1);
      if (!product && !flat) return false;
      any = true;
    }
    if ((e.sym == S_MEMOFFSET || e.sym == S_MALLOC) && overlaps(e.out, e.out_bytes, p, bytes)) return any;
    if ((e.sym == S_DEALLOC && e.out == p) || e.sym == S_POOLFREE) return any;
    if (e.sym == S_OPAQUE) return false;
    if (e.sym != S_MEMOFFSET && e.sym != S_MALLOC && e.out && overlaps(e.out, e.out_bytes, p, bytes)) return false;
  }
  return false;
}

// The first reader of [p, p+bytes) from entry `from` on when all readers are convolutions of the 16-bit
// path with this tensor as their input (one only, if it has the few channels of a stem); -1 otherwise.
int only_convs_read(const std::vector<Entry> &rec, uintptr_t p, int64_t bytes, size_t from) {
  int first = -1;
  for (size_t t = from; t < rec.size(); ++t) {
    const Entry &e = rec[t];
    for (int k = 0; k < 3; ++k) {
      if (!e.in[k] || !overlaps(e.in[k], e.in_bytes[k] > 0 ? e.in_bytes[k] : 1, p, bytes)) continue;
      if (k != 0 || (e.sym != S_CONV && e.sym != S_CONV_BIAS_ACT) || e.in[0] != p || e.in_bytes[0] != bytes ||
          !entry_reads_16(e))
        return -1;
      const bool few = e.args.v[1] < 16;
      if (first >= 0 && (few || rec[first].args.v[1] < 16)) return -1;
      if (first < 0) first = (int)t;
    }
    if ((e.sym == S_MEMOFFSET || e.sym == S_MALLOC) && overlaps(e.out, e.out_bytes, p, bytes)) return first;
    if ((e.sym == S_DEALLOC && e.out == p) || e.sym == S_POOLFREE) return first;
    if (e.sym == S_OPAQUE) return -1;
    if (e.sym != S_MEMOFFSET && e.sym != S_MALLOC && e.out && overlaps(e.out, e.out_bytes, p, bytes)) return -1;
  }
  return -1;
}

// True when everything that reads [p, p+bytes) from entry `from` on, until the range is handed out again
// or freed, takes fp32 values in three planes: dense convolutions of fp32 mode, sums folded into one,
// pools and means.
bool only_parts_read(const std::vector<Entry> &rec, const std::vector<uint16_t> &roles, uintptr_t p, int64_t bytes,
                     size_t from) {
  bool any = false;
  for (size_t t = from; t < rec.size(); ++t) {
    const Entry &e = rec[t];
    for (int k = 0; k < 3; ++k) {
      if (!e.in[k] || !overlaps(e.in[k], e.in_bytes[k] > 0 ? e.in_bytes[k] : 1, p, bytes)) continue;
      if (e.in[k] != p || e.in_bytes[k] != bytes) return false;
      const bool conv = (e.sym == S_CONV || e.sym == S_CONV_BIAS_ACT) && k == 0 && e.parts;
      const bool sum = e.sym == S_TENSOR_OP && e.kind == CK_SAME_ADD && (roles[t] & ROLE_BITS) == R_ABSORB;
      const bool pool = e.sym == S_MAXPOOL || e.sym == S_AVGPOOL || e.sym == S_REDUCE;
      if (!conv && !sum && !pool) return false;
      any = true;
    }
    if ((e.sym == S_MEMOFFSET || e.sym == S_MALLOC) && overlaps(e.out, e.out_bytes, p, bytes)) return any;
    if ((e.sym == S_DEALLOC && e.out == p) || e.sym == S_POOLFREE) return any;
    if (e.sym == S_OPAQUE) return false;
    if (any && e.out == p && e.out_bytes == bytes) return true;
    if (e.sym != S_MEMOFFSET && e.sym != S_MALLOC && e.out && overlaps(e.out, e.out_bytes, p, bytes)) return false;
  }
  return false;
}

// Marks the chains of a finished inference: R_DEFER on the convolution, R_ABSORB on the
// calls folded into it.
void analyse(const std::vector<Entry> &rec, std::vector<uint16_t> &roles, std::vector<int> &reader) {
  roles.assign(rec.size(), R_EAGER);
  reader.assign(rec.size(), -1);
  // of every convolution: the last call folded into it, and the tensor that one writes
  std::vector<size_t> chain_last(rec.size(), 0);
  std::vector<uintptr_t> chain_out(rec.size(), 0);
  std::vector<bool> chain_res(rec.size(), false), chain_act(rec.size(), false);
  std::vector<size_t> chain_add(rec.size(), 0);   // the sum with another tensor
  for (size_t i = 0; i < rec.size(); ++i) {
    const Entry &c = rec[i];
    if (c.sym == S_D2D && (reader[i] = only_convs_read(rec, c.out, c.out_bytes, i + 1)) >= 0)
      roles[i] |= RF_FOR_CONV;
    if ((c.sym == S_REDUCE || c.sym == S_AVGPOOL || c.sym == S_MAXPOOL) && c.out != c.in[0] &&
        only_matmuls_read(rec, c.out, c.out_bytes, i + 1))
      roles[i] |= RF_FOR_MATMUL;
    if (c.sym == S_MATMUL && c.fusable) {
      // product -> bias row (in place or not) -> ReLU
      bool bias_set = false, act_set = false;
      uintptr_t cur = c.out;
      size_t last = i;
      std::vector<size_t> members;
      for (size_t j = i + 1; j < rec.size() && !act_set; ++j) {
        const Entry &f = rec[j];
        if (is_passive(f.sym)) {
          if ((f.sym == S_MEMOFFSET || f.sym == S_MALLOC) && overlaps(f.out, f.out_bytes, cur, c.out_bytes)) break;
          if (f.sym == S_DEALLOC && f.out == cur) break;
          continue;
        }
        const bool shape = f.dims[0] == c.dims[0] && f.dims[1] == c.dims[1] && f.out_bytes == c.out_bytes;
        const bool take = shape && f.in[0] == cur &&
                          ((f.sym == S_TENSOR_OP && f.kind == CK_ROW_BIAS && !bias_set) ||
                           (f.sym == S_ACTIVE && f.kind == CK_RELU));
        if (!take) break;
        if (f.out != cur && !dies_unread(rec, cur, c.out_bytes, j + 1)) break;
        if (f.sym == S_TENSOR_OP) bias_set = true;
        else act_set = true;
        members.push_back(j);
        last = j;
        cur = f.out;
      }
      if (!members.empty()) {
        roles[i] |= R_DEFER;
        for (size_t m : members) roles[m] |= R_ABSORB;
      }
      if (only_matmuls_read(rec, cur, c.out_bytes, last + 1)) {
        roles[i] |= RF_FOR_MATMUL;   // on the product, for the chain as a whole
      }
      continue;
    }
    if ((c.sym != S_CONV && c.sym != S_CONV_BIAS_ACT) || !c.fusable) continue;
    bool bias_set = c.sym == S_CONV_BIAS_ACT;
    bool act_set = c.sym == S_CONV_BIAS_ACT && c.kind != 5;
    bool res_set = false;
    uintptr_t cur = c.out;
    const int64_t cur_bytes = c.out_bytes;
    std::vector<size_t> members;
    for (size_t j = i + 1; j < rec.size() && !act_set; ++j) {
      const Entry &f = rec[j];
      if (is_passive(f.sym)) {
        // the chain's running tensor must stay in place until it is consumed
        if ((f.sym == S_MEMOFFSET || f.sym == S_MALLOC) && overlaps(f.out, f.out_bytes, cur, cur_bytes))
          break;
        if (f.sym == S_DEALLOC && f.out == cur) break;
        continue;
      }
      bool take = false;
      if (f.sym == S_TENSOR_OP && f.kind == CK_BIAS_ADD && f.in[0] == cur && !bias_set && !res_set &&
          same_dims(f, c)) {
        take = true;
      } else if (f.sym == S_TENSOR_OP && f.kind == CK_SAME_ADD && !res_set && !c.depthwise &&
                 ((f.in[0] == cur) != (f.in[1] == cur)) && same_dims(f, c)) {
        take = true;
      } else if ((f.sym == S_ACTIVE && f.kind == CK_RELU) || (f.sym == S_CLIP && f.kind == CK_CLIP)) {
        take = f.in[0] == cur && same_dims(f, c);
      }
      if (!take) break;
      // skipping the write of `cur` is allowed only if this call was its sole reader
      if (f.out != cur && !dies_unread(rec, cur, cur_bytes, j + 1)) break;
      if (f.sym == S_TENSOR_OP && f.kind == CK_BIAS_ADD) bias_set = true;
      else if (f.sym == S_TENSOR_OP) res_set = true, chain_add[i] = j;
      else act_set = true;
      members.push_back(j);
      cur = f.out;
    }
    // a stem convolution takes the max pool behind it along, some others a 2x2 one, when the pool is the
    // only reader of the full-resolution tensor
    if (!res_set && !c.depthwise && !c.parts) {
      const size_t from = members.empty() ? i + 1 : members.back() + 1;
      for (size_t j = from; j < rec.size(); ++j) {
        const Entry &f = rec[j];
        if (is_passive(f.sym)) {
          if ((f.sym == S_MEMOFFSET || f.sym == S_MALLOC) && overlaps(f.out, f.out_bytes, cur, cur_bytes))
            break;
          if (f.sym == S_DEALLOC && f.out == cur) break;
          continue;
        }
        if (f.sym == S_MAXPOOL && f.in[0] == cur && f.out != cur && dies_unread(rec, cur, cur_bytes, j + 1) &&
            ((c.poolable && f.kind == CK_POOL_3S2) || (f.kind == CK_POOL_2S2 && entry_takes_pool(c))))
          members.push_back(j);
        break;
      }
    }
    chain_last[i] = members.empty() ? i : members.back();
    chain_out[i] = cur;
    chain_res[i] = res_set;
    chain_act[i] = act_set;
    if (members.empty()) continue;
    roles[i] |= R_DEFER;
    for (size_t m : members) roles[m] |= R_ABSORB;
  }
  // Inverted residuals: a 1x1 convolution whose result only a 3x3 depthwise one reads, whose result only
  // another 1x1 one reads.
  auto next_alone = [&](size_t i) -> size_t {   // the convolution that alone reads the chain of `i`, or 0
    const uintptr_t cur = chain_out[i];
    const int64_t bytes = rec[i].out_bytes;
    for (size_t j = chain_last[i] + 1; j < rec.size(); ++j) {
      const Entry &f = rec[j];
      if (is_passive(f.sym)) {
        if ((f.sym == S_MEMOFFSET || f.sym == S_MALLOC) && overlaps(f.out, f.out_bytes, cur, bytes)) return 0;
        if (f.sym == S_DEALLOC && f.out == cur) return 0;
        continue;
      }
      const bool conv = (f.sym == S_CONV || f.sym == S_CONV_BIAS_ACT) && f.fusable && !f.parts && f.in[0] == cur &&
                        f.in_bytes[0] == bytes && f.in[1] != cur;
      return conv && dies_unread(rec, cur, bytes, j + 1) ? j : 0;
    }
    return 0;
  };
  auto one_by_one = [](const Entry &e) {
    const int64_t *v = e.args.v;   // dX[4], dW[4], pads[2], strides[2], groups
    return !e.depthwise && v[6] == 1 && v[7] == 1 && v[8] == 0 && v[9] == 0 && v[10] == 1 && v[11] == 1 && v[12] == 1;
  };
  for (size_t i = 0; i < rec.size(); ++i) {
    const Entry &a = rec[i];
    if ((a.sym != S_CONV && a.sym != S_CONV_BIAS_ACT) || !a.fusable || a.parts || !one_by_one(a) || chain_res[i])
      continue;
    const size_t j = next_alone(i);
    if (!j) continue;
    const int64_t *w = rec[j].args.v;
    if (!rec[j].depthwise || w[6] != 3 || w[7] != 3 || w[8] != 1 || w[9] != 1 || w[10] != w[11] || chain_res[j]) continue;
    const size_t k = next_alone(j);
    if (!k || !one_by_one(rec[k])) continue;
    const int64_t *v = a.args.v;
    if (!ir_supported((int)v[0], (int)v[1], (int)v[4], (int)rec[k].args.v[4], (int)v[2], (int)v[3],
                      (int)rec[k].dims[2], (int)rec[k].dims[3], (int)w[10], mode_f16()))
      continue;
    roles[i] = (uint16_t)(R_DEFER | RF_LINK);
    roles[j] = (uint16_t)(R_DEFER | RF_LINK | RF_JOIN);
    roles[k] = (uint16_t)(R_DEFER | RF_JOIN);
  }
  // Sums of two convolutions: the chain in front of one that ends in a sum is the other summand, nobody else
  // reads it, and nothing but constants arriving lies between the two.
  auto passive_past = [&](size_t from, size_t to, uintptr_t p, int64_t bytes) {   // [p, p+bytes) stays what it is
    for (size_t t = from; t < to; ++t) {
      const Entry &e = rec[t];
      if (!is_passive(e.sym)) return false;
      if (e.out && overlaps(e.out, e.out_bytes > 0 ? e.out_bytes : 1, p, bytes)) return false;
    }
    return true;
  };
  for (size_t i = 1; i < rec.size(); ++i) {
    if (!chain_res[i]) continue;
    const Entry &b = rec[i], &add = rec[chain_add[i]];
    size_t a = i;
    while (a > 0 && !((rec[a - 1].sym == S_CONV || rec[a - 1].sym == S_CONV_BIAS_ACT) && rec[a - 1].fusable)) --a;
    if (a-- == 0) continue;
    const Entry &c = rec[a];
    const uintptr_t sum = chain_out[a];
    if (c.depthwise || b.depthwise || c.parts || b.parts || chain_res[a] || chain_act[a] || !same_dims(c, b) ||
        ((roles[a] | roles[i]) & (RF_LINK | RF_JOIN)) || !sum || (add.in[0] != sum && add.in[1] != sum) ||
        !passive_past(chain_last[a] + 1, i, sum, c.out_bytes))
      continue;
    bool ok = true;
    for (size_t t = i; t < chain_add[i] && ok; ++t) {   // the second chain up to the sum
      const Entry &e = rec[t];
      if (is_passive(e.sym)) ok = passive_past(t, t + 1, sum, c.out_bytes);
      else if (overlaps(e.out, e.out_bytes, sum, c.out_bytes)) ok = false;
      for (int k = 0; k < 3; ++k)
        if (e.in[k] && overlaps(e.in[k], e.in_bytes[k] > 0 ? e.in_bytes[k] : 1, sum, c.out_bytes)) ok = false;
    }
    if (!ok || (add.out != sum && !dies_unread(rec, sum, c.out_bytes, chain_add[i] + 1))) continue;
    roles[a] = (uint16_t)((roles[a] & ~ROLE_BITS) | R_DEFER | RF_SUM);
    roles[i] |= RF_SUM;
  }
  // A block's last convolution and the next block's first.
  for (size_t i = 0; i < rec.size(); ++i) {
    const Entry &c = rec[i];
    if (!chain_res[i] || !chain_act[i] || c.depthwise || c.parts || (roles[i] & (RF_LINK | RF_JOIN)) || c.dims[1] % 128)
      continue;
    size_t j = chain_last[i] + 1;
    while (j < rec.size() && is_passive(rec[j].sym)) ++j;
    if (j == rec.size() || (rec[j].sym != S_CONV && rec[j].sym != S_CONV_BIAS_ACT)) continue;
    const Entry &f = rec[j];
    if (!f.fusable || f.parts || !one_by_one(f) || f.in[0] != chain_out[i] || f.in_bytes[0] != c.out_bytes || chain_res[j] ||
        !chain_act[j] || (roles[j] & (RF_LINK | RF_JOIN | RF_SUM)) || !passive_past(chain_last[i] + 1, j, chain_out[i], c.out_bytes))
      continue;
    // The first result is written when both chains are complete: its place must not be handed out again before that.
    bool stays = true;
    for (size_t t = j; t <= chain_last[j] && stays; ++t)
      stays = !is_passive(rec[t].sym) || passive_past(t, t + 1, chain_out[i], c.out_bytes);
    if (!stays) continue;
    roles[i] |= RF_LEAD;
    roles[j] = (uint16_t)((roles[j] & ~ROLE_BITS) | R_DEFER | RF_FOLLOW);
  }
  for (size_t i = 0; i < rec.size(); ++i)   // (after the roles are known)
    if ((rec[i].parts || (roles[i] & ROLE_BITS) == R_ABSORB) &&
        only_parts_read(rec, roles, rec[i].out, rec[i].out_bytes, i + 1))
      roles[i] |= RF_FOR_PARTS;
}

// Writes the adopted prefix out as calls of this inference, their pointers moved to its pool.
void trace_rewind_entries() {
  TraceState &ts = g_ts;
  if (!ts.prefix_len) return;
  std::vector<Entry> all(ts.prefix->entries.begin(), ts.prefix->entries.begin() + ts.prefix_len);
  const uintptr_t from = ts.prefix->pool_base, bytes = ts.prefix->pool_bytes, to = ts.last_pool_base;
  auto move = [&](uintptr_t a) { return a >= from && a < from + bytes ? a - from + to : a; };
  for (Entry &e : all) {
    for (int k = 0; k < 3; ++k) e.in[k] = move(e.in[k]);
    e.out = move(e.out);
    for (int k = 0; k < 4; ++k) e.args.p[k] = (void *)move((uintptr_t)e.args.p[k]);
  }
  all.insert(all.end(), ts.rec.begin(), ts.rec.end());
  ts.rec.swap(all);
  ts.prefix = nullptr;
  ts.prefix_len = 0;
}

}  // namespace

bool trace_enabled() {
  if (g_ts.enabled < 0) {
    const char *e = getenv("OCCAMY_FUSE_ACROSS_CALLS");
    g_ts.enabled = (e && !strcmp(e, "0")) ? 0 : 1;
  }
  return g_ts.enabled == 1;
}

void trace_set_enabled(bool on) {
  g_ts.enabled = on ? 1 : 0;
  if (!on) {
    g_ts.programs.clear();
    g_ts.cands.clear();
    g_ts.rec.clear();
    g_ts.prefix = nullptr;
    g_ts.prefix_len = 0;
    g_ts.in_inference = false;
  }
}

Entry trace_entry(int sym) {
  Entry e;
  e.sym = sym;
  mix(e.sig, (uint64_t)sym);
  return e;
}

void te_ptr(Entry &e, const void *p) {
  uintptr_t a = (uintptr_t)p;
  if (g_ts.pool_base && a >= g_ts.pool_base && a < g_ts.pool_base + g_ts.pool_bytes)
    a = (a - g_ts.pool_base) | (1ull << 63);
  mix(e.sig, (uint64_t)a);
}
void te_ptr_or_elsewhere(Entry &e, const void *p) {
  uintptr_t a = (uintptr_t)p;
  const bool inside = a >= g_ts.pool_base && a < g_ts.pool_base + g_ts.pool_bytes;
  if (!g_ts.pool_base || inside || reg_find(p)) te_ptr(e, p);
  else mix(e.sig, 1);
}
void te_i(Entry &e, int64_t v) { mix(e.sig, (uint64_t)v); }
void te_f(Entry &e, float v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  mix(e.sig, u);
}
void te_dims(Entry &e, const int64_t *d, int n) {
  for (int i = 0; i < n; ++i) mix(e.sig, (uint64_t)d[i]);
}

void trace_force(uint16_t role) { g_ts.forced = role; }
void trace_force_end() { g_ts.forced = -1; }

Role trace_step(Entry &e, bool *deviated) {
  *deviated = false;
  TraceState &ts = g_ts;
  ts.last_flags = 0;
  if (ts.forced >= 0) {
    ts.last_flags = (uint16_t)(ts.forced & ~ROLE_BITS);
    return (Role)(ts.forced & ROLE_BITS);
  }
  if (!trace_enabled() || !ts.in_inference) return R_EAGER;
  if (trace_index() >= MAX_ENTRIES) {  // not a compiled model's call pattern: stop tracing
    ts.in_inference = false;
    *deviated = ts.matched_so_far;
    ts.matched_so_far = false;
    return R_EAGER;
  }
  const size_t index = trace_index();
  ts.last_flags = 0;
  Role role = R_EAGER;
  if (!ts.cands.empty()) {
    size_t keep = 0;
    for (size_t k = 0; k < ts.cands.size(); ++k) {
      const TraceProgram &p = ts.programs[ts.cands[k]];
      if (index < p.sigs.size() && p.sigs[index] == e.sig) ts.cands[keep++] = ts.cands[k];
    }
    ts.cands.resize(keep);
    if (keep) {
      // recorded programs that share this prefix must agree on the call's role (two models
      // with the same first layers may continue differently); otherwise it runs as it stands.  What
      // it does together with the convolution behind or before it is left out if they disagree on that alone.
      uint16_t r = ts.programs[ts.cands[0]].roles[index];
      for (size_t k = 1; k < keep; ++k)
        r &= ~((r ^ ts.programs[ts.cands[k]].roles[index]) & RF_TOGETHER);
      role = (Role)(r & ROLE_BITS);
      ts.last_flags = r & (uint16_t)~ROLE_BITS;
      for (size_t k = 1; k < keep; ++k)
        if (((ts.programs[ts.cands[k]].roles[index] ^ r) & ~RF_TOGETHER) ||
            ((r & RF_FOR_CONV) && ts.programs[ts.cands[k]].sigs[ts.programs[ts.cands[k]].reader[index]] !=
                                      ts.programs[ts.cands[0]].sigs[ts.programs[ts.cands[0]].reader[index]])) {
          role = R_EAGER;
          ts.last_flags = 0;
        }
      ts.matched_so_far = true;
    } else {
      *deviated = ts.matched_so_far;
      ts.matched_so_far = false;
    }
  }
  ts.rec.push_back(e);
  return role;
}

void trace_begin() {
  TraceState &ts = g_ts;
  if (!trace_enabled()) return;
  ts.in_inference = true;
  ts.matched_so_far = false;
  ts.rec.clear();
  ts.prefix = nullptr;
  ts.prefix_len = 0;
  ts.elided = 0;
  ts.last_pool_base = ts.pool_base;   // a pool set up before cudnnCreate; otherwise none yet
  ts.last_pool_bytes = ts.pool_bytes;
  ts.cands.clear();
  for (size_t i = 0; i < ts.programs.size(); ++i) ts.cands.push_back((int)i);
}

void trace_end() {
  TraceState &ts = g_ts;
  if (!trace_enabled() || !ts.in_inference) return;
  ts.in_inference = false;
  const size_t n = trace_index();
  bool known = false;
  for (int c : ts.cands)
    if (ts.programs[c].sigs.size() == n) known = true;
  if (!known && n) {
    trace_rewind_entries();
    TraceProgram p;
    p.sigs.reserve(n);
    for (const Entry &e : ts.rec) p.sigs.push_back(e.sig);
    analyse(ts.rec, p.roles, p.reader);
    p.entries.swap(ts.rec);
    p.pool_base = ts.last_pool_base;
    p.pool_bytes = ts.last_pool_bytes;
    if (ts.programs.size() >= MAX_PROGRAMS) ts.programs.erase(ts.programs.begin());
    ts.programs.push_back(std::move(p));
  }
  ts.rec.clear();
  ts.prefix = nullptr;
  ts.prefix_len = 0;
  ts.cands.clear();
}

// ---- prefixes made in one go (graph_replay.cu) ------------------------------------
uint16_t trace_last_flags() { return g_ts.last_flags; }
const Entry *trace_last_reader() {
  TraceProgram *p = g_ts.cands.empty() ? nullptr : &g_ts.programs[g_ts.cands[0]];
  const size_t n = trace_index();
  if (!p || !n || n > p->reader.size() || p->reader[n - 1] < 0) return nullptr;
  return &p->entries[p->reader[n - 1]];
}
bool trace_active() { return trace_enabled() && g_ts.in_inference; }
size_t trace_index() { return g_ts.prefix_len + g_ts.rec.size(); }
TraceProgram *trace_candidate() {
  return g_ts.cands.size() == 1 ? &g_ts.programs[g_ts.cands[0]] : nullptr;
}
void trace_mark_uploaded() {
  if (trace_active() && !g_ts.rec.empty()) g_ts.rec.back().uploaded = true;
}
bool trace_has_own_entries() { return g_ts.prefix_len == 0; }
const std::vector<Entry> &trace_entries() { return g_ts.rec; }
uintptr_t trace_pool_base() { return g_ts.pool_base; }
size_t trace_pool_bytes() { return g_ts.pool_bytes; }

void trace_adopt_prefix(TraceProgram *p, size_t n) {
  g_ts.rec.clear();
  g_ts.prefix = p;
  g_ts.prefix_len = n;
}

void trace_rewind(TraceProgram *p, size_t n) {
  TraceState &ts = g_ts;
  trace_adopt_prefix(p, n);
  trace_rewind_entries();
  ts.cands.clear();
  for (size_t i = 0; i < ts.programs.size(); ++i) {
    const TraceProgram &q = ts.programs[i];
    if (q.sigs.size() >= n && std::equal(q.sigs.begin(), q.sigs.begin() + n, p->sigs.begin()))
      ts.cands.push_back((int)i);
  }
  ts.matched_so_far = true;
}

void trace_set_pool(void *base, size_t bytes) {
  g_ts.pool_base = (uintptr_t)base;
  g_ts.pool_bytes = bytes;
  if (base) {
    g_ts.last_pool_base = (uintptr_t)base;
    g_ts.last_pool_bytes = bytes;
  }
}

void trace_note_elided() {
  g_ts.elided++;
}
bool trace_has_elided() { return g_ts.elided > 0; }
int64_t trace_fused_chains() { return g_ts.fused_chains; }
void trace_count_chain() { g_ts.fused_chains++; }

}  // namespace occ
