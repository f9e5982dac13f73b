// Tapes: the calls of one run, kept so that a later run of the same shapes is one call of the host.
//
// Between wdc_tape_begin and wdc_tape_end every entry point notes itself (WDC_TAPE, below): the function, its scalars
// and descriptors by value, and each device pointer as "offset into the n-th buffer of the run" when it lies in an
// input or in something the run allocated, else as the address itself (weights and other data that outlive the run).
// wdc_alloc and wdc_free are noted too.  wdc_tape_run then repeats the calls with new buffers.
#pragma once

#include <functional>
#include <map>
#include <new>
#include <tuple>
#include <utility>
#include <vector>

#include "common.cuh"

struct wdc_tape {
  struct Ref {
    int slot = -1;          // buffer of the run, or -1: `base` is the address
    int64_t offset = 0;
    char* base = nullptr;
    char* at(char* const* slots) const { return slot < 0 ? base : slots[slot] + offset; }
  };
  typedef std::function<int(wdc_context*, char**)> Op;
  std::vector<Op> ops;
  int n_in = 0, n_slots = 0;
  std::vector<int64_t> in_bytes;
  std::vector<int> outs;    // slots of the run's results
  // while recording
  wdc_context* ctx = nullptr;
  int depth = 0;            // entry points call one another: only the outermost is noted
  bool valid = true;
  std::map<char*, std::pair<int, int64_t>> live;   // base -> (slot, bytes)

  Ref ref(const void* p) const {
    Ref r;
    r.base = (char*)p;
    auto it = live.upper_bound((char*)p);
    if (p && it != live.begin()) {
      --it;
      if ((char*)p < it->first + it->second.second) {
        r.slot = it->second.first;
        r.offset = (char*)p - it->first;
      }
    }
    return r;
  }
};

// The tape this thread is recording (only its own calls belong to the run), or null.
extern thread_local wdc_tape* wdc_thread_tape;

// Brackets an entry point; `tape` is set when the call is the outermost one of a recording.
struct TapeScope {
  wdc_tape* counted = nullptr;
  wdc_tape* tape = nullptr;
  explicit TapeScope(wdc_context* ctx) {
    wdc_tape* t = wdc_thread_tape;
    if (!t || t->ctx != ctx) return;
    counted = t;
    if (t->depth++ == 0) tape = t;
  }
  ~TapeScope() {
    if (counted) counted->depth--;
  }
};

// How an argument is kept.  Pointers are device pointers unless wrapped in tape_desc / tape_array.
template <class T>
struct TapeArg {
  T v;
  TapeArg(const wdc_tape&, T a) : v(a) {}
  T get(char* const*) const { return v; }
};
template <class T>
struct TapeArg<T*> {
  wdc_tape::Ref r;
  TapeArg(const wdc_tape& t, T* a) : r(t.ref((const void*)a)) {}
  T* get(char* const* slots) const { return (T*)r.at(slots); }
};
template <class D>
struct TapeDesc {
  D d{};
};
template <class D>
TapeDesc<D> tape_desc(const D* d) {
  TapeDesc<D> t;
  if (d) t.d = *d;
  return t;
}
template <class D>
struct TapeArg<TapeDesc<D>> {
  D d;
  TapeArg(const wdc_tape&, const TapeDesc<D>& a) : d(a.d) {}
  const D* get(char* const*) const { return &d; }
};
struct TapeArray {
  int64_t v[6] = {};
};
inline TapeArray tape_array(const int64_t* p, int n) {
  TapeArray t;
  for (int i = 0; p && i < n && i < 6; i++) t.v[i] = p[i];
  return t;
}
template <>
struct TapeArg<TapeArray> {
  TapeArray a;
  TapeArg(const wdc_tape&, const TapeArray& x) : a(x) {}
  const int64_t* get(char* const*) const { return a.v; }
};

template <class F, class Kept, size_t... I>
int tape_call(F fn, const Kept& kept, wdc_context* ctx, char** slots, std::index_sequence<I...>) {
  return fn(ctx, std::get<I>(kept).get(slots)...);
}
// (the entry points are C: a tape that does not fit in memory is given up)
template <class F, class... A>
void tape_note(wdc_tape* t, F fn, A... args) {
  typedef std::tuple<TapeArg<A>...> Kept;
  try {
    const Kept kept{TapeArg<A>(*t, args)...};
    t->ops.push_back([fn, kept](wdc_context* ctx, char** slots) {
      return tape_call(fn, kept, ctx, slots, std::make_index_sequence<sizeof...(A)>());
    });
  } catch (const std::bad_alloc&) {
    t->valid = false;
  }
}

// First statement of an entry point behind its null check.
#define WDC_TAPE(ctx, fn, ...)  \
  TapeScope tape_scope_(ctx);   \
  if (tape_scope_.tape) tape_note(tape_scope_.tape, fn, __VA_ARGS__)
// An entry point whose call cannot be repeated (it moves host data, waits, or changes the context).
#define WDC_NO_TAPE(ctx)       \
  TapeScope tape_scope_(ctx);  \
  if (tape_scope_.tape) tape_scope_.tape->valid = false

// A captured run (context.cu).
struct wdc_graph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  wdc_arena* arena = nullptr;  // owns every buffer the captured launches touch that was allocated while capturing
  // The recorded launches hold the addresses of the tensor-core path's cached operand splits (hi/lo copies of
  // the weights).  split_seq = the context's split counter when the capture ended: if a split that is that old
  // is dropped later (its weight was rewritten or freed), the graph would read freed memory, so it goes stale.
  int64_t split_seq = 0;
  bool stale = false;
  // wdc_graph_run with small transfers: the graph between one kernel that brings the inputs in from page-locked memory
  // (index 1; index 0 leaves that out) and one that takes the outputs there, so that a run is one launch and one wait
  cudaGraphExec_t io_exec[2] = {nullptr, nullptr};
  bool io_failed = false;
  char* io_host = nullptr;          // page-locked: inputs, then outputs
  int64_t io_in_bytes = 0, io_bytes = 0;
  wdc_io_list io_in[2] = {}, io_out = {};   // what the kernels were made with
  std::mutex io_mu;                 // a run owns the staging memory from its inputs to its outputs
};
