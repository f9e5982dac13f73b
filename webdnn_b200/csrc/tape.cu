// Recording and repeating the calls of a run (see tape.cuh), and a captured graph's run with its host transfers.
#include <string.h>

#include <memory>

#include "tape.cuh"

thread_local wdc_tape* wdc_thread_tape = nullptr;

extern "C" int wdc_tape_begin(wdc_context* ctx, int n_in, void* const* in, const int64_t* bytes) {
  if (!ctx || n_in < 0 || (n_in > 0 && (!in || !bytes)))
    return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_begin: bad argument");
  if (wdc_thread_tape) return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_begin: this thread is already recording a tape");
  if (ctx->capture_arena) return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_begin: a capture is open");
  wdc_tape* t = new (std::nothrow) wdc_tape();
  if (!t) return wdc_fail(ctx, WDC_ERR_OOM, "wdc_tape_begin: out of host memory");
  t->ctx = ctx;
  t->n_in = t->n_slots = n_in;
  try {
    for (int i = 0; i < n_in; i++) {
      t->in_bytes.push_back(bytes[i]);
      // (an input passed twice, or an empty one, could not be told from its twin)
      if (in[i] && bytes[i] > 0) t->valid &= t->live.insert({(char*)in[i], {i, bytes[i]}}).second;
    }
  } catch (const std::bad_alloc&) {
    delete t;
    return wdc_fail(ctx, WDC_ERR_OOM, "wdc_tape_begin: out of host memory");
  }
  wdc_thread_tape = t;
  return WDC_OK;
}

void wdc_tape_forget(wdc_context* ctx) {
  if (!wdc_thread_tape || wdc_thread_tape->ctx != ctx) return;
  delete wdc_thread_tape;
  wdc_thread_tape = nullptr;
}

extern "C" int wdc_tape_end(wdc_context* ctx, int n_out, void* const* out, wdc_tape** tape) {
  if (!ctx || !tape || (n_out > 0 && !out)) return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_end: bad argument");
  *tape = nullptr;
  wdc_tape* t = wdc_thread_tape;
  if (!t || t->ctx != ctx) return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_end: no tape is being recorded");
  wdc_thread_tape = nullptr;
  // every result is a buffer of its own that the run allocated, and nothing else it allocated is left
  size_t left = 0;
  for (auto& kv : t->live)
    if (kv.second.first >= t->n_in) left++;
  try {
    std::vector<bool> taken((size_t)t->n_slots, false);
    for (int i = 0; i < n_out && t->valid; i++) {
      const wdc_tape::Ref r = t->ref(out[i]);
      t->valid = r.slot >= t->n_in && r.offset == 0 && !taken[(size_t)r.slot];
      if (t->valid) {
        taken[(size_t)r.slot] = true;
        t->outs.push_back(r.slot);
      }
    }
  } catch (const std::bad_alloc&) {
    t->valid = false;
  }
  if (n_out < 0 || left != (size_t)n_out) t->valid = false;
  t->live.clear();
  if (!t->valid) {
    delete t;
    return WDC_OK;
  }
  *tape = t;
  return WDC_OK;
}

extern "C" int wdc_tape_destroy(wdc_context* ctx, wdc_tape* tape) {
  if (!ctx) return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_destroy: null context");
  delete tape;
  return WDC_OK;
}

// What wdc_alloc and wdc_free note about themselves.
void wdc_tape_note_alloc(wdc_tape* t, void* p, int64_t bytes) {
  const int slot = t->n_slots++;
  try {
    t->live[(char*)p] = {slot, bytes > 0 ? bytes : 1};
    t->ops.push_back([slot, bytes](wdc_context* ctx, char** slots) {
      return wdc_alloc(ctx, bytes, (void**)&slots[slot]);
    });
  } catch (const std::bad_alloc&) {
    t->valid = false;
  }
}
void wdc_tape_note_free(wdc_tape* t, void* p) {
  auto it = t->live.find((char*)p);
  if (it == t->live.end()) {   // not the run's own buffer
    t->valid = false;
    return;
  }
  const int slot = it->second.first;
  const bool input = slot < t->n_in;
  t->live.erase(it);
  try {
    t->ops.push_back([slot, input](wdc_context* ctx, char** slots) {
      // an input is the run's own where it came from host memory: the caller keeps its device buffers
      if (input && !slots[-1 - slot]) return (int)WDC_OK;
      void* q = slots[slot];
      slots[slot] = nullptr;
      return wdc_free(ctx, q);
    });
  } catch (const std::bad_alloc&) {
    t->valid = false;
  }
}

extern "C" int wdc_tape_run(wdc_context* ctx, wdc_tape* tape, const void* const* in, const int32_t* in_on_host,
                            void** out, void* const* out_host, const int64_t* out_bytes) {
  if (!ctx || !tape || (tape->n_in > 0 && (!in || !in_on_host)) || (!tape->outs.empty() && !out))
    return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_tape_run: bad argument");
  WDC_NO_TAPE(ctx);
  DeviceGuard g(ctx->device);
  // (in front of the slots, from the last one back: whether an input's buffer is the run's own)
  std::unique_ptr<char*[]> buffers(new (std::nothrow) char*[(size_t)(tape->n_in + tape->n_slots)]());
  if (!buffers) return wdc_fail(ctx, WDC_ERR_OOM, "wdc_tape_run: out of host memory");
  char** const slots = buffers.get() + tape->n_in;
  int s = WDC_OK;
  for (int i = 0; i < tape->n_in && s == WDC_OK; i++) {
    if (!in_on_host[i]) {
      slots[i] = (char*)in[i];
      continue;
    }
    s = wdc_alloc(ctx, tape->in_bytes[(size_t)i], (void**)&slots[i]);
    slots[-1 - i] = slots[i];
    if (s == WDC_OK && tape->in_bytes[(size_t)i] > 0) s = wdc_stage_in(ctx, slots[i], in[i], tape->in_bytes[(size_t)i]);
  }
  for (size_t k = 0; k < tape->ops.size() && s == WDC_OK; k++) s = tape->ops[k](ctx, slots);
  for (int i = 0; i < tape->n_in; i++)   // stream-ordered: reused only by work queued after this run
    if (in_on_host[i] && slots[i]) {
      wdc_free(ctx, slots[i]);
      slots[i] = nullptr;
    }
  const int n_out = (int)tape->outs.size();
  if (s == WDC_OK) {
    for (int i = 0; i < n_out; i++) out[i] = slots[tape->outs[(size_t)i]];
    if (!out_host) return WDC_OK;
    s = wdc_stage_out(ctx, n_out, out_host, (const void* const*)out, out_bytes);
  }
  // results have been read, or a call failed: nothing of the run stays allocated
  for (int i = tape->n_in; i < tape->n_slots; i++)
    if (slots[i]) wdc_free(ctx, slots[i]);
  for (int i = 0; i < n_out; i++) out[i] = nullptr;
  return s;
}

namespace {

constexpr int64_t IO_LIMIT = 128 << 10;   // transfers that a kernel makes (see transfer.cu)

int64_t padded(int64_t bytes) { return bytes > 0 ? (bytes + 15) / 16 * 16 : 0; }

// The graph with its transfers as kernels at both ends (`with_in`: inputs too).  Null when it could not be made.
cudaGraphExec_t io_graph(wdc_graph* g, bool with_in, const wdc_io_list& in, const wdc_io_list& out) {
  if (g->io_exec[with_in])   // (made for other buffers: the caller goes the general way)
    return g->io_in[with_in] == in && g->io_out == out ? g->io_exec[with_in] : nullptr;
  if (g->io_failed || (g->io_exec[!with_in] && !(g->io_out == out))) return nullptr;
  cudaGraph_t whole = nullptr;
  cudaGraphNode_t first = nullptr, body = nullptr, last = nullptr;
  auto kernel_node = [](const wdc_io_list& list, void** args) {
    cudaKernelNodeParams k = {};
    k.func = wdc_io_kernel();
    k.gridDim = wdc_io_grid(list);
    k.blockDim = dim3(256);
    k.kernelParams = args;
    return k;
  };
  wdc_io_list in_copy = in, out_copy = out;
  void* in_args[] = {&in_copy};
  void* out_args[] = {&out_copy};
  cudaError_t e = cudaGraphCreate(&whole, 0);
  if (e == cudaSuccess && with_in) {
    const cudaKernelNodeParams k = kernel_node(in, in_args);
    e = cudaGraphAddKernelNode(&first, whole, nullptr, 0, &k);
  }
  if (e == cudaSuccess) e = cudaGraphAddChildGraphNode(&body, whole, first ? &first : nullptr, first ? 1 : 0, g->graph);
  if (e == cudaSuccess) {
    const cudaKernelNodeParams k = kernel_node(out, out_args);
    e = cudaGraphAddKernelNode(&last, whole, &body, 1, &k);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&g->io_exec[with_in], whole, 0);
  if (whole) cudaGraphDestroy(whole);
  if (e != cudaSuccess) {
    cudaGetLastError();
    g->io_failed = true;
    g->io_exec[with_in] = nullptr;
  }
  g->io_in[with_in] = in;
  g->io_out = out;
  return g->io_exec[with_in];
}

// A run whose outputs (and, when they come from the host, inputs) are small.  False: not taken, nothing happened.
bool run_small(wdc_context* ctx, wdc_graph* g, int n_in, void* const* dst, const void* const* src, const int64_t* in_bytes,
               const int32_t* in_on_host, int n_out, void* const* host, const void* const* out, const int64_t* out_bytes,
               int* status) {
  int64_t in_total = 0, out_total = 0;
  bool from_host = n_in > 0, words = true;
  for (int i = 0; i < n_in; i++) {
    in_total += padded(in_bytes[i]);
    from_host &= in_on_host[i] != 0;
    words &= in_bytes[i] % 4 == 0;
  }
  for (int i = 0; i < n_out; i++) {
    out_total += padded(out_bytes[i]);
    words &= out_bytes[i] % 4 == 0;
  }
  if (g->stale || g->io_failed || ctx->capture_arena || !words || n_out < 1 || n_out > wdc_io_list::MOST ||
      n_in > wdc_io_list::MOST || out_total > IO_LIMIT || out_total == 0)
    return false;
  const bool with_in = from_host && in_total > 0 && in_total <= IO_LIMIT;
  std::lock_guard<std::mutex> lk(g->io_mu);
  if (!g->io_host) {   // (sized by the first run; the buffers of a captured run do not change)
    g->io_bytes = (in_total <= IO_LIMIT ? in_total : 0) + out_total;
    g->io_in_bytes = in_total <= IO_LIMIT ? in_total : 0;
    if (cudaMallocHost((void**)&g->io_host, (size_t)g->io_bytes) != cudaSuccess) {
      cudaGetLastError();
      g->io_failed = true;
      return false;
    }
  }
  if ((with_in && in_total != g->io_in_bytes) || g->io_in_bytes + out_total > g->io_bytes) return false;
  wdc_io_list ins = {}, outs = {};
  int64_t at = 0;
  for (int i = 0; with_in && i < n_in; i++) {
    if (in_bytes[i] <= 0) continue;
    memcpy(g->io_host + at, src[i], (size_t)in_bytes[i]);
    ins.part[ins.n++] = {(uint32_t*)dst[i], (const uint32_t*)(g->io_host + at), in_bytes[i] / 4};
    at += padded(in_bytes[i]);
  }
  at = g->io_in_bytes;
  for (int i = 0; i < n_out; i++) {
    if (out_bytes[i] <= 0) continue;
    outs.part[outs.n++] = {(uint32_t*)(g->io_host + at), (const uint32_t*)out[i], out_bytes[i] / 4};
    at += padded(out_bytes[i]);
  }
  cudaGraphExec_t exec = io_graph(g, with_in, ins, outs);
  if (!exec) return false;
  int s = WDC_OK;
  for (int i = 0; i < n_in && s == WDC_OK; i++) {
    if (in_bytes[i] <= 0) continue;
    wdc_tc_evict(ctx, dst[i], in_bytes[i]);
    if (with_in) ctx->h2d_bytes += in_bytes[i];
    else if (in_on_host[i]) s = wdc_stage_in(ctx, dst[i], src[i], in_bytes[i]);
    else
      s = wdc_check_cuda(ctx, cudaMemcpyAsync(dst[i], src[i], (size_t)in_bytes[i], cudaMemcpyDeviceToDevice, ctx->stream),
                         "copy of an input");
  }
  if (s == WDC_OK && g->stale) s = wdc_graph_launch(ctx, g);   // (gone stale just now: the error it gives)
  else if (s == WDC_OK) {
    s = wdc_check_cuda(ctx, cudaGraphLaunch(exec, ctx->stream), "cudaGraphLaunch");
    ctx->n_launch++;
  }
  if (s == WDC_OK) s = wdc_sync(ctx);
  for (int i = 0, k = 0; i < n_out && s == WDC_OK; i++) {
    if (out_bytes[i] <= 0) continue;
    memcpy(host[i], outs.part[k++].dst, (size_t)out_bytes[i]);
    ctx->d2h_bytes += out_bytes[i];
  }
  *status = s;
  return true;
}

}  // namespace

extern "C" int wdc_graph_run(wdc_context* ctx, wdc_graph* graph, int n_in, void* const* dst, const void* const* src,
                             const int64_t* in_bytes, const int32_t* in_on_host, int n_out, void* const* host,
                             const void* const* out, const int64_t* out_bytes) {
  if (!ctx || !graph || n_in < 0 || n_out < 0 || (n_in > 0 && (!dst || !src || !in_bytes || !in_on_host)) ||
      (n_out > 0 && (!host || !out || !out_bytes)))
    return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_graph_run: bad argument");
  WDC_NO_TAPE(ctx);
  DeviceGuard g(ctx->device);
  int small = WDC_OK;
  if (run_small(ctx, graph, n_in, dst, src, in_bytes, in_on_host, n_out, host, out, out_bytes, &small)) return small;
  for (int i = 0; i < n_in; i++) {
    if (in_bytes[i] <= 0) continue;
    wdc_tc_evict(ctx, dst[i], in_bytes[i]);
    if (in_on_host[i]) {
      const int s = wdc_stage_in(ctx, dst[i], src[i], in_bytes[i]);
      if (s != WDC_OK) return s;
    } else {
      WDC_CUDA(ctx, cudaMemcpyAsync(dst[i], src[i], (size_t)in_bytes[i], cudaMemcpyDeviceToDevice, ctx->stream));
    }
  }
  const int s = wdc_graph_launch(ctx, graph);
  if (s != WDC_OK) return s;
  return n_out > 0 ? wdc_stage_out(ctx, n_out, host, out, out_bytes) : WDC_OK;
}
