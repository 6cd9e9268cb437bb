// Recorded inferences as CUDA graphs.
//
// A compiled model makes the same few hundred runtime calls for every inference, and making them -
// signatures, format registry, tensor maps, some sixty launches - took 300 to 400 us of host time,
// more than the GPU needs for a small batch.  Once an inference has run call by call with nothing
// left to upload or allocate, its calls from the one after the input's arrival up to the last
// computing one (the window) are recorded as graphs; later inferences only check that each call
// is the recorded one (signature, and for a constant its host address and fingerprint) and the
// graphs are launched in its place, each as soon as the last of its calls has come by.
//
// A call that differs - another shape, a changed constant, anything outside the window - takes the
// inference back: the calls that no launched graph covers are made again one by one, then the
// differing one as it stands.
#pragma once
#include <functional>

#include "runtime.h"
#include "trace.h"

namespace occ {

// Start of a traced call.  True: the call is covered by a graph and must do nothing but return.
bool graph_covers(const Entry &e);
// End of a call that was carried out.
void graph_after_call();
// Something is about to happen that calls held back must come before (another entry point waits for
// the stream, reads a result, changes a mode): everything up to here is enqueued.
void graph_settle();
// Work that cannot be recorded follows (an allocation, a packing, a wait): what has been recorded is
// launched, the rest of the inference is not recorded.
void graph_stop_capture();
// The same for an upload, which the trace notes as well: a window does not reach across it.
void graph_before_upload();
// An upload of `bytes` to `dst`, recorded just now, is about to start; `copy_stream` waits for what may still use that
// memory.  When the inference's window exists cut up by images, the upload is made in as many pieces on
// `copy_stream`, and true is returned: the window takes the pieces as they arrive, and any other call waits for the
// last.
bool graph_upload_in_pieces(void *dst, const void *src, size_t bytes, cudaStream_t copy_stream);
// Device memory that graphs may refer to is about to be freed or its contents replaced.
void graph_forget_all();
// A call is about to be carried out that no graph covers.
void graph_uncovered();
// This call is not the recorded one, and may read any tensor: a window computed in pieces, which left nothing but its
// result, is made call by call.
void graph_left_recording();
// Frees what windows cut up by images work in.
void graph_free_memory();
// cudnnCreate / cudnnDestroy.
void graph_inference_begin();
void graph_inference_end();

// abi.cu: makes a recorded call again.
void run_again(const Entry &e, const std::function<void *(void *)> &place, const void *host);
// abi.cu: enqueues a held-back convolution; whether there is one.
void flush_held_back();
bool anything_held_back();

}  // namespace occ
