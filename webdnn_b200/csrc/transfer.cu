// Transfers between host and device memory on the compute stream.
//
// The driver moves pageable memory through its own staging buffers with one thread: 11 us for 4 KB before anything
// else can be queued, 12.7 GB/s for megabytes (605 us for an 800x800 image), where the link takes 50 GB/s from
// page-locked memory.  Here the context keeps a ring of page-locked chunks: a transfer is cut into chunks, each is
// copied by a few threads and sent (or received and copied) while its neighbours are on the link.  Page-locked
// buffers of the caller's go straight to the link.  Small results leave the copy engines out: a kernel of the compute
// stream writes the page-locked memory, which saves the switch between the two.
#include <sched.h>
#include <string.h>

#include <atomic>
#include <condition_variable>
#include <exception>
#include <new>
#include <thread>

#include "tape.cuh"

namespace {

constexpr int64_t CHUNK = 512 << 10;    // long enough to hide an event and a copy call (a few us) behind 10 us of link
constexpr int CHUNKS = 32;
constexpr int64_t PIECE = 64 << 10;     // what a thread takes at a time
constexpr int64_t ALONE = 256 << 10;    // below this the other threads would only be woken up
constexpr int64_t PINNED_CHECK = 256 << 10;   // asking the driver what a pointer is costs about a microsecond
constexpr int64_t BY_KERNEL = 128 << 10;      // up to here the link's latency, not its rate, is the time
constexpr int MAX_HELPERS = 5;

// CPUs this process may run on, and the helpers of all its contexts: together they stay below that number.
int usable_cpus() {
  cpu_set_t set;
  CPU_ZERO(&set);
  if (sched_getaffinity(0, sizeof(set), &set) == 0 && CPU_COUNT(&set) > 0) return CPU_COUNT(&set);
  const unsigned n = std::thread::hardware_concurrency();
  return n > 0 ? (int)n : 1;
}
std::atomic<int> helpers_alive{0};

// memcpy by the caller and up to MAX_HELPERS threads that take pieces from a common counter: a helper that is still
// asleep costs nothing, the caller takes its pieces (all of them where no thread could be had).  Helpers poll for a while
// after a job, then sleep.
class CopyTeam {
 public:
  ~CopyTeam() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : helpers_) t.join();
    helpers_alive.fetch_sub((int)helpers_.size());
  }
  // dst[c] <- src in chunks of CHUNK bytes; sent(c) is called by the caller's thread, in order, as chunks are complete.
  template <class F>
  void copy(char* const* dst, const char* src, int64_t bytes, F sent) {
    const int chunks = (int)((bytes + CHUNK - 1) / CHUNK);
    if (bytes < ALONE) {
      memcpy(dst[0], src, (size_t)bytes);
      sent(0);
      return;
    }
    if (!started_) start();
    Job job;
    job.dst = dst;
    job.src = src;
    job.bytes = bytes;
    job.pieces = (int)((bytes + PIECE - 1) / PIECE);
    {
      std::lock_guard<std::mutex> lk(mu_);
      job_ = &job;
      seq_.fetch_add(1, std::memory_order_release);
    }
    if (asleep_.load() > 0) cv_.notify_all();
    for (int c = 0; c < chunks;) {
      const int64_t n = bytes - (int64_t)c * CHUNK < CHUNK ? bytes - (int64_t)c * CHUNK : CHUNK;
      if (job.done[c].load(std::memory_order_acquire) == (int)((n + PIECE - 1) / PIECE)) sent(c++);
      else if (!take(job)) pause();
    }
    {
      std::lock_guard<std::mutex> lk(mu_);   // no helper picks the job up any more ...
      job_ = nullptr;
    }
    while (job.users.load(std::memory_order_acquire) > 0) pause();   // ... and those who did have left it
  }
  void copy(char* dst, const char* src, int64_t bytes) {   // at most one chunk
    copy(&dst, src, bytes, [](int) {});
  }

 private:
  struct Job {
    char* const* dst;
    const char* src;
    int64_t bytes;
    int pieces;
    std::atomic<int> next{0}, users{0};
    std::atomic<int> done[CHUNKS] = {};   // pieces of a chunk that have been copied
  };
  static void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
  }
  // Copies the next piece; false when none is left.
  static bool take(Job& j) {
    const int i = j.next.fetch_add(1, std::memory_order_relaxed);
    if (i >= j.pieces) return false;
    const int64_t off = (int64_t)i * PIECE, n = j.bytes - off < PIECE ? j.bytes - off : PIECE;
    memcpy(j.dst[off / CHUNK] + off % CHUNK, j.src + off, (size_t)n);
    j.done[off / CHUNK].fetch_add(1, std::memory_order_release);
    return true;
  }
  void start() {
    started_ = true;
    const int most = usable_cpus() - 1;
    for (int i = 0; i < MAX_HELPERS; i++) {
      bool made = false;
      if (helpers_alive.fetch_add(1) < most) {
        try {
          helpers_.emplace_back([this] { run(); });
          made = true;
        } catch (const std::exception&) {   // no thread to be had
        }
      }
      if (!made) {
        helpers_alive.fetch_sub(1);
        return;
      }
    }
  }
  void run() {
    uint64_t seen = 0;
    for (;;) {
      int polls = 0;
      while (seq_.load(std::memory_order_acquire) == seen && polls < 20000) {   // some 0.5 ms
        pause();
        polls++;
      }
      Job* job = nullptr;
      {
        std::unique_lock<std::mutex> lk(mu_);
        if (seq_.load() == seen) {
          asleep_++;
          cv_.wait(lk, [&] { return stop_ || seq_.load() != seen; });
          asleep_--;
        }
        if (stop_) return;
        seen = seq_.load();
        job = job_;
        if (job) job->users.fetch_add(1, std::memory_order_relaxed);
      }
      if (job) {
        while (take(*job)) {}
        job->users.fetch_sub(1, std::memory_order_release);
      }
    }
  }
  std::vector<std::thread> helpers_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<uint64_t> seq_{0};
  std::atomic<int> asleep_{0};
  Job* job_ = nullptr;
  bool started_ = false, stop_ = false;
};

}  // namespace

struct wdc_stager {
  std::mutex mu;             // one transfer at a time uses the ring
  char* ring = nullptr;
  cudaEvent_t done[CHUNKS] = {};
  bool busy[CHUNKS] = {};    // a transfer recorded done[i] and nobody has waited for it yet
  int next = 0;
  CopyTeam team;
};

namespace {

void stager_free(wdc_stager* s) {
  for (auto& ev : s->done)
    if (ev) cudaEventDestroy(ev);
  if (s->ring) cudaFreeHost(s->ring);
  delete s;
}

int stager_of(wdc_context* ctx, wdc_stager** out) {
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (!ctx->stager) {
    wdc_stager* s = new (std::nothrow) wdc_stager();
    if (!s) return wdc_fail(ctx, WDC_ERR_OOM, "page-locked staging memory: out of host memory");
    cudaError_t e = cudaMallocHost((void**)&s->ring, (size_t)(CHUNKS * CHUNK));
    for (auto& ev : s->done)
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (e != cudaSuccess) {   // the next transfer tries again
      cudaGetLastError();
      stager_free(s);
      return wdc_check_cuda(ctx, e, "page-locked staging memory");
    }
    ctx->stager = s;
  }
  *out = ctx->stager;
  return WDC_OK;
}

// The next chunk of the ring, free for use.
int take_chunk(wdc_context* ctx, wdc_stager* s, int* index) {
  const int i = s->next;
  s->next = (i + 1) % CHUNKS;
  if (s->busy[i]) {
    WDC_CUDA(ctx, cudaEventSynchronize(s->done[i]));
    s->busy[i] = false;
  }
  *index = i;
  return WDC_OK;
}

bool page_locked(const void* p, int64_t bytes) {
  if (bytes < PINNED_CHECK) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

// Words of several buffers, copied by one launch.  Page-locked host memory on one side.
__global__ void __launch_bounds__(256) io_copy_kernel(const wdc_io_list list) {
  for (int s = 0; s < list.n; s++) {
    const wdc_io_list::Part p = list.part[s];
    const int64_t vec = (((uintptr_t)p.dst | (uintptr_t)p.src) & 15) == 0 ? p.words / 4 : 0;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = first; i < vec; i += step)
      reinterpret_cast<uint4*>(p.dst)[i] = __ldcv(reinterpret_cast<const uint4*>(p.src) + i);
    for (int64_t i = vec * 4 + first; i < p.words; i += step) p.dst[i] = __ldcv(p.src + i);
  }
}

}  // namespace

dim3 wdc_io_grid(const wdc_io_list& list) {
  int64_t most = 0;
  for (int i = 0; i < list.n; i++) most = list.part[i].words > most ? list.part[i].words : most;
  const int64_t blocks = ceil_div64(most, 4 * 256);
  return dim3((unsigned)(blocks < 1 ? 1 : blocks < 64 ? blocks : 64));
}
void* wdc_io_kernel() { return (void*)io_copy_kernel; }

void wdc_stager_destroy(wdc_context* ctx) {
  if (ctx->stager) stager_free(ctx->stager);
  ctx->stager = nullptr;
}

// host -> device, ordered with the compute stream; pageable sources may be released when the call returns.
int wdc_stage_in(wdc_context* ctx, void* dst, const void* host, int64_t bytes) {
  if (ctx->capture_arena)
    return wdc_fail(ctx, WDC_ERR_INVALID, "a transfer from host memory cannot be part of a captured run");
  ctx->h2d_bytes += bytes;
  if (page_locked(host, bytes)) {
    WDC_CUDA(ctx, cudaMemcpyAsync(dst, host, (size_t)bytes, cudaMemcpyHostToDevice, ctx->stream));
    return WDC_OK;
  }
  wdc_stager* s = nullptr;
  int st = stager_of(ctx, &s);
  if (st != WDC_OK) return st;
  std::lock_guard<std::mutex> lk(s->mu);
  for (int64_t base = 0; base < bytes; base += CHUNKS * CHUNK) {   // a ring's worth at a time
    const int64_t part = bytes - base < CHUNKS * CHUNK ? bytes - base : CHUNKS * CHUNK;
    int index[CHUNKS];
    char* chunk[CHUNKS];
    for (int64_t off = 0; off < part; off += CHUNK) {
      const int c = (int)(off / CHUNK);
      st = take_chunk(ctx, s, &index[c]);
      if (st != WDC_OK) return st;
      chunk[c] = s->ring + index[c] * CHUNK;
    }
    cudaError_t e = cudaSuccess;
    s->team.copy(chunk, (const char*)host + base, part, [&](int c) {
      const int64_t off = (int64_t)c * CHUNK, n = part - off < CHUNK ? part - off : CHUNK;
      if (e == cudaSuccess)
        e = cudaMemcpyAsync((char*)dst + base + off, chunk[c], (size_t)n, cudaMemcpyHostToDevice, ctx->stream);
      if (e == cudaSuccess) e = cudaEventRecord(s->done[index[c]], ctx->stream);
      if (e == cudaSuccess) s->busy[index[c]] = true;
    });
    if (e != cudaSuccess) return wdc_check_cuda(ctx, e, "transfer to the device");
  }
  return WDC_OK;
}

// device -> host for several buffers; waits for the compute stream.
int wdc_stage_out(wdc_context* ctx, int count, void* const* host, const void* const* src, const int64_t* bytes) {
  if (ctx->capture_arena)
    return wdc_fail(ctx, WDC_ERR_INVALID, "a transfer to host memory cannot be part of a captured run");
  wdc_stager* s = nullptr;
  int st = stager_of(ctx, &s);
  if (st != WDC_OK) return st;
  int64_t total = 0;
  bool words = true;
  for (int b = 0; b < count; b++) {
    total += bytes[b] > 0 ? (bytes[b] + 15) / 16 * 16 : 0;
    words &= bytes[b] % 4 == 0;
  }
  if (total > 0 && total <= BY_KERNEL && words && count <= wdc_io_list::MOST) {
    std::lock_guard<std::mutex> lk(s->mu);
    int i;
    st = take_chunk(ctx, s, &i);
    if (st != WDC_OK) return st;
    char* at = s->ring + i * CHUNK;
    wdc_io_list list = {};
    for (int b = 0; b < count; b++) {
      if (bytes[b] <= 0) continue;
      ctx->d2h_bytes += bytes[b];
      list.part[list.n++] = {(uint32_t*)at, (const uint32_t*)src[b], bytes[b] / 4};
      at += (bytes[b] + 15) / 16 * 16;
    }
    io_copy_kernel<<<wdc_io_grid(list), 256, 0, ctx->stream>>>(list);
    WDC_CUDA(ctx, cudaGetLastError());
    st = wdc_sync(ctx);
    if (st != WDC_OK) return st;
    for (int b = 0, k = 0; b < count; b++)
      if (bytes[b] > 0) memcpy(host[b], list.part[k++].dst, (size_t)bytes[b]);
    return WDC_OK;
  }
  {
    std::lock_guard<std::mutex> lk(s->mu);
    struct Part {
      char* to;
      int64_t n;
      int chunk;
    };
    Part queue[CHUNKS];
    int head = 0, queued = 0;
    auto finish_one = [&]() -> int {
      Part& p = queue[head];
      head = (head + 1) % CHUNKS;
      queued--;
      WDC_CUDA(ctx, cudaEventSynchronize(s->done[p.chunk]));
      s->busy[p.chunk] = false;
      s->team.copy(p.to, s->ring + p.chunk * CHUNK, p.n);
      return WDC_OK;
    };
    for (int b = 0; b < count; b++) {
      if (bytes[b] <= 0) continue;
      ctx->d2h_bytes += bytes[b];
      if (page_locked(host[b], bytes[b])) {
        WDC_CUDA(ctx, cudaMemcpyAsync(host[b], src[b], (size_t)bytes[b], cudaMemcpyDeviceToHost, ctx->stream));
        continue;
      }
      for (int64_t off = 0; off < bytes[b]; off += CHUNK) {
        const int64_t n = bytes[b] - off < CHUNK ? bytes[b] - off : CHUNK;
        if (queued == CHUNKS) {
          st = finish_one();
          if (st != WDC_OK) return st;
        }
        int i;
        st = take_chunk(ctx, s, &i);
        if (st != WDC_OK) return st;
        WDC_CUDA(ctx, cudaMemcpyAsync(s->ring + i * CHUNK, (const char*)src[b] + off, (size_t)n, cudaMemcpyDeviceToHost,
                                      ctx->stream));
        WDC_CUDA(ctx, cudaEventRecord(s->done[i], ctx->stream));
        s->busy[i] = true;
        queue[(head + queued) % CHUNKS] = {(char*)host[b] + off, n, i};
        queued++;
      }
    }
    while (queued) {
      st = finish_one();
      if (st != WDC_OK) return st;
    }
  }
  return wdc_sync(ctx);
}

extern "C" int wdc_upload(wdc_context* ctx, void* dst, const void* host, int64_t bytes) {
  if (!ctx || bytes < 0 || (bytes > 0 && (!dst || !host)))
    return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_upload: bad argument");
  WDC_NO_TAPE(ctx);
  if (bytes == 0) return WDC_OK;
  DeviceGuard g(ctx->device);
  wdc_tc_evict(ctx, dst, bytes);
  return wdc_stage_in(ctx, dst, host, bytes);
}

extern "C" int wdc_download(wdc_context* ctx, void* host, const void* src, int64_t bytes) {
  if (!ctx || bytes < 0 || (bytes > 0 && (!host || !src)))
    return wdc_fail(ctx, WDC_ERR_INVALID, "wdc_download: bad argument");
  WDC_NO_TAPE(ctx);
  DeviceGuard g(ctx->device);
  return wdc_stage_out(ctx, 1, &host, &src, &bytes);
}
