// Call trace of one inference and the plan derived from it.
//
// A model compiled by Occamy is straight-line code: every inference issues the same
// runtime calls with the same shapes and the same pool offsets.  The runtime records the
// calls between cudnnCreate and cudnnDestroy (the compiled function's prologue and
// epilogue).  When an inference ends it looks for chains
//     convolution -> [+ bias [1,K,1,1]] -> [+ same-shape tensor] -> [ReLU | Clip]
//     matrix product -> [+ bias row] -> [ReLU]
//     1x1 convolution chain -> 3x3 depthwise chain -> 1x1 convolution chain
//     convolution chain + convolution chain [-> ReLU | Clip]
//     convolution chain with a sum and ReLU -> 1x1 convolution chain with ReLU, both of whose results are kept
// (and, for a few-channel stem convolution, a 3x3 / stride 2 max pool behind it)
// whose intermediate results nobody else reads before their memory is handed out again,
// and marks them.  The next time the same call sequence comes by, the convolution of such
// a chain is held back, the following calls are folded into its epilogue, and one kernel
// writes only the chain's final tensor.  A call that does not match the recorded sequence
// ends the speculation: whatever is held back is executed as it stands.
#pragma once
#include <cstddef>
#include <cstdint>
#include <memory>
#include <vector>

namespace occ {

enum Sym {
  S_POOLINIT = 1, S_MEMOFFSET, S_MALLOC, S_H2D, S_D2H, S_D2D, S_DEALLOC, S_POOLFREE,
  S_CONV, S_CONV_BIAS_ACT, S_TENSOR_OP, S_ACTIVE, S_CLIP, S_MAXPOOL, S_AVGPOOL, S_REDUCE,
  S_MATMUL, S_SOFTMAX, S_FLATTEN, S_RESHAPE, S_OPAQUE
};

// R_SKIP: the call is part of a recorded stretch that runs as one CUDA graph (graph_replay.h)
enum Role { R_EAGER = 0, R_DEFER = 1, R_ABSORB = 2, R_SKIP = 3 };

// kind of a tensor-op / activation entry, as far as chains care
enum ChainKind {
  CK_NONE = 0, CK_BIAS_ADD = 1, CK_SAME_ADD = 2, CK_RELU = 3, CK_CLIP = 4,
  CK_POOL_3S2 = 5,  // max pool 3x3, stride 2, pad 1
  CK_ROW_BIAS = 6,  // rank 2: the same row added to every row
  CK_POOL_2S2 = 7   // max pool 2x2, stride 2, no padding
};

// The call's own arguments, enough to make it again (graph_replay.cu, run_again).
struct CallArgs {
  void *p[4] = {nullptr, nullptr, nullptr, nullptr};
  int64_t v[24] = {};
  float f[2] = {0.f, 0.f};
  bool whole = true;   // all of them (the dimensions of a call may be more than fit)
};

struct Entry {
  uint64_t sig = 1469598103934665603ull;
  int sym = 0;
  uintptr_t in[3] = {0, 0, 0};
  int64_t in_bytes[3] = {0, 0, 0};   // fp32 extent of each input (0: unknown, taken as one byte)
  uintptr_t out = 0;
  int64_t out_bytes = 0;   // fp32 extent of `out` (range size for the memory calls)
  int64_t dims[4] = {0, 0, 0, 0};
  int kind = CK_NONE;      // ChainKind, or the activation mode of a fused convolution
  bool fusable = false;    // convolution or product that the tensor cores take (may head a chain)
  bool parts = false;      // ... in fp32 mode: operands as bf16 parts of fp32 values
  bool depthwise = false;
  bool poolable = false;   // convolution whose kernel can take a following CK_POOL_3S2 along
  bool uploaded = false;   // S_H2D: bytes crossed to the device (not a constant that is already there)
  const void *host = nullptr;   // S_H2D: source
  CallArgs args;
};

// Signature building.  Device pointers are taken relative to the active pool when they
// lie inside it; host pointers are left out of signatures.
Entry trace_entry(int sym);
void te_ptr(Entry &e, const void *p);
void te_i(Entry &e, int64_t v);
void te_f(Entry &e, float v);
void te_dims(Entry &e, const int64_t *d, int n);

// The same for a copy's other end: while a pool is active, any device address that is no tensor of the runtime's
// counts as "elsewhere" (the caller's batch, its result buffer).
void te_ptr_or_elsewhere(Entry &e, const void *p);

// A recorded inference: the calls between cudnnCreate and cudnnDestroy and the role of each.
struct GraphPlan;
// flag beside a call's role: whatever reads its result is a matrix product (possibly behind a Flatten),
// so the result may be kept in the 16-bit form that product takes
constexpr uint16_t RF_FOR_MATMUL = 0x10;
// on a device-to-device copy: what reads the tensor are convolutions on the 16-bit path, so the copy may
// bring it in in their form (TraceProgram::reader names the first of them)
constexpr uint16_t RF_FOR_CONV = 0x20;
// on a convolution in fp32 mode or a call folded into one: all that reads the result takes it in three
// planes of parts (FMT_PARTS)
constexpr uint16_t RF_FOR_PARTS = 0x40;
// on convolutions that run together with the next one (RF_LINK) or the one before (RF_JOIN): the three of
// an inverted residual, which become one kernel
constexpr uint16_t RF_LINK = 0x04;
constexpr uint16_t RF_JOIN = 0x08;
// on two convolutions whose results are added, one chain behind the other: the first is held back until the sum
// comes by, which one kernel then computes (a block's last convolution and its projection shortcut)
constexpr uint16_t RF_SUM = 0x80;
// on a convolution whose chain ends in a sum and ReLU, and on the 1x1 convolution right behind it that reads the
// result: one kernel may write both (launch_tc_pair())
constexpr uint16_t RF_LEAD = 0x100;
constexpr uint16_t RF_FOLLOW = 0x200;
constexpr uint16_t RF_TOGETHER = RF_SUM | RF_LEAD | RF_FOLLOW;   // each may be left out
constexpr uint16_t ROLE_BITS = 0x03;
struct TraceProgram {
  std::vector<uint64_t> sigs;
  std::vector<uint16_t> roles;   // Role | RF_*
  std::vector<int> reader;      // RF_FOR_CONV: call that reads the result first
  std::vector<Entry> entries;
  uintptr_t pool_base = 0;     // pool the entries' pointers refer to
  size_t pool_bytes = 0;
  std::shared_ptr<GraphPlan> graph;
};

// Records the call and returns the role the matching recorded program gives it.
// *deviated is set when this call is the first of the inference that matches no recorded
// program although earlier calls did.
Role trace_step(Entry &e, bool *deviated);

uint16_t trace_last_flags();        // RF_* of the call trace_step() was last given
const Entry *trace_last_reader();   // the recorded call that first reads its result (RF_FOR_CONV)
void trace_begin();                 // cudnnCreate
void trace_end();                   // cudnnDestroy: analyse and store if the sequence is new
// ---- for graph_replay.cu ----
bool trace_active();                // between the two, and tracing
size_t trace_index();               // calls of this inference so far
TraceProgram *trace_candidate();    // the one recorded program that matches so far, or null
void trace_mark_uploaded();         // the call recorded last moved bytes to the device
bool trace_has_own_entries();       // this inference was recorded call by call
const std::vector<Entry> &trace_entries();
// The calls up to `n` are those of `p`, made without trace_step().
void trace_adopt_prefix(TraceProgram *p, size_t n);
// The same, as if they had been made one by one: what follows is recorded and matched anew.
void trace_rewind(TraceProgram *p, size_t n);
// (abi.cu) whether the convolution's kernel can take a following CK_POOL_2S2 along; whether it reads its input
// as a 16-bit tensor
bool entry_takes_pool(const Entry &e);
bool entry_reads_16(const Entry &e);
// The role (with its RF_*) of the calls up to trace_force_end(), whatever was recorded: calls made outside an
// inference's own sequence.
void trace_force(uint16_t role);
void trace_force_end();
uintptr_t trace_pool_base();
size_t trace_pool_bytes();
void trace_set_pool(void *base, size_t bytes);
void trace_note_elided();           // a tensor of this inference was skipped by a fusion
bool trace_has_elided();
bool trace_enabled();
void trace_set_enabled(bool on);   // turning it off also forgets the recorded programs
int64_t trace_fused_chains();       // chains executed fused since load
void trace_count_chain();

}  // namespace occ
