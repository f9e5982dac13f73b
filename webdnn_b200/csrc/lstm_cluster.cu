// ONNX LSTM recurrence on the 5th-generation tensor cores, spread over the chip as thread-block clusters: hidden sizes whose R
// does not fit one cluster (above 512; lstm_local.cu has the others, 2.4 us a step of [64, 512] where this takes 3.3).
//
// What bounds a recurrence is the chain of one step, not its arithmetic: h_t cannot start before h_{t-1} is known
// everywhere.  lstm_persistent.cu spends 9 us on a step of [64, 512]: every CTA waits for a counter that all CTAs
// bump, brings the whole h_{t-1} in (128 KB each), and 2 us of FMAs follow.  This kernel shortens every link:
//   * A cluster owns 32 hidden units (128 gate rows = the 128 TMEM lanes of an MMA); its CTAs split K.  A CTA's slice
//     of R stays in TENSOR MEMORY for the whole sequence (A operand, high and low TF32 parts), so a step's product
//     is a few dozen tcgen05.mma of M 128 x N batch x K 8 against the CTA's slice of h_{t-1} in shared memory.
//   * Only that slice is read, not all of h.  There is no counter and no fence: Y is filled with a NaN pattern that
//     arithmetic cannot produce before the launch, h_t is written straight into Y[t], and a reader polls the words
//     it needs until none of them is the pattern.  The exchange between clusters is one store and one load.
//   * The partial sums of the K slices meet through distributed shared memory: each CTA finishes 32 / CS units, and
//     every thread sends its columns with st.async to the CTA that finishes its row, whose mbarrier counts the bytes.
//     Two buffers and two barriers, by the parity of the step: a CTA reaches step t + 2 only after every CTA of the
//     cluster has sent step t + 1, i.e. has read step t.
// Measured: a step of [1, 544] 2.0 us, of [64, 544] 5.0 (two groups of rows fit the GPU), of [1,
// 768] 2.2, of [64, 768] 5.8 (one group).
// All clusters of a launch wait for one another, so the launch is cooperative (all resident or an error).
// Products are 3xTF32 with rounded parts (2^-23 of a product), sums fp32; gates as in lstm_persistent.cu.  An infinite
// element of R or h0 would meet low parts of either sign or zero: a CTA whose slice holds one sums with plain fp32 FMAs.
// Waits are bounded (2 s): on expiry the CTA sets the context's status word and leaves at its next barrier; its
// peers' waits expire in turn, and all meet at a last cluster barrier, so no CTA leaves while others may write to it.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int THREADS = 256;
constexpr int UNITS = 32;             // units of a cluster: 4 gate rows each
constexpr int CS = 4;                 // CTAs of a cluster (17 clusters of 8, for the first size that gets here, do not fit the GPU)
constexpr int UPC = UNITS / CS;       // units a CTA finishes
constexpr int ROWS = 4 * UPC;         // their gate rows
constexpr int PAIRS = 4;              // (unit, batch row) pairs a thread finishes, at most
constexpr int D_COLS = 128;           // TMEM columns of the accumulator (batch rows of a launch, at most)
constexpr int KC_MAX = (512 - D_COLS) / 2;   // K slice: high and low parts of R fill the rest of tensor memory
constexpr int MAX_ITEMS = 12;         // 16-byte words of h a thread brings in per step, at most
constexpr int MAX_SMEM = 226 * 1024;
constexpr uint32_t EMPTY = 0xffffffffu;   // not yet written; arithmetic gives 0x7fffffff for every NaN
constexpr unsigned long long WAIT_NS = 2000000000ull;

struct ClusterArgs {
  const float* P;      // [T, B, 4H] input projection without bias
  const float* R;      // [4H, H]
  const float* bias;   // [8H] or null
  const float* h0;     // [B, H] or null
  const float* c0;
  float* Y;            // [T, B, H], filled with EMPTY
  float* Yh;
  float* Yc;
  int* status;
  int T, B, H;
  int b0, nb;          // this launch handles batch rows b0 .. b0 + nb - 1 ...
  int per;             // ... in groups of `per` rows, each on clusters of its own
  int n;               // per rounded up to 16: columns of the MMA
  int kc;              // K slice of a CTA of a cluster (a multiple of 8)
  int blocks;          // clusters of a group: ceil(H / 32)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, int* status, int code) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 256; i++)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > WAIT_NS) {
      atomicCAS(status, 0, code);
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, int code) {
  for (int i = 0; i < 1024; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, status, code);
}
__device__ __forceinline__ uint4 ld_relaxed(const float* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ bool is_empty(const uint4& v) {
  return v.x == EMPTY || v.y == EMPTY || v.z == EMPTY || v.w == EMPTY;
}
__device__ __forceinline__ uint32_t map_to(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send16(uint32_t dst, uint32_t bar, const float* v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// x = high + low with the high part rounded to TF32 (11 bits) and the low part exact before the tensor core cuts it
__device__ __forceinline__ float high_part(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {   // K-major, 128B swizzle
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D += A * B with the shared-memory descriptor as its two halves: only the low one (the start address) changes from
// MMA to MMA, and the single issuing lane's instructions are on the chain of a step.
template <bool kAccumulate>
__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_c, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi,
                                             uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 d;\n\t"
      "mov.b64 d, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], d, %4, p;\n\t}"
      :
      : "r"(tmem_c), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
// One k step: lo*hi + hi*lo + hi*hi
template <bool kFirst>
__device__ __forceinline__ void umma_step(uint32_t tmem_c, uint32_t a_hi, uint32_t a_lo, uint32_t d_hi, uint32_t d_lo,
                                          uint32_t desc_top, uint32_t idesc) {
  umma_tf32_ts<!kFirst>(tmem_c, a_lo, d_hi, desc_top, idesc);
  umma_tf32_ts<true>(tmem_c, a_hi, d_lo, desc_top, idesc);
  umma_tf32_ts<true>(tmem_c, a_hi, d_hi, desc_top, idesc);
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float* v) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ float sigmoid_ref(float x) { return (tanhf(x * 0.5f) + 1.f) * 0.5f; }

struct ClusterShared {
  unsigned long long mma_bar;
  unsigned long long recv_bar[2];
  unsigned int tmem_base;
  int abort;
  int plain_r, plain_h;     // R's slice, or h0's, holds an element whose high part is not finite
};

// A step's sums of gate row `row` and `cols` batch rows from c0 on without the tensor cores, sent like the accumulator's.
// h: the slice of h_{t-1} in global memory (null: zero); rows past nb are not used by anyone.
__device__ __noinline__ void send_plain_sums(const float* R, const float* h, int H, int nb, int c0, int cols, int u0, int row, int k0,
                                             int klen, uint32_t dst, uint32_t dst_step, uint32_t bar) {
  const int unit = u0 + row / 4;
  const float* r = R + ((size_t)(row & 3) * H + (unit < H ? unit : 0)) * H + k0;
  for (int c = c0; c < c0 + cols; c += 4, dst += dst_step) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int q = 0; q < 4 && unit < H && c + q < nb; q++) {
      for (int k = 0; k < klen; k++) {
        float x = 0.f;
        if (h) asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(x) : "l"(h + (size_t)(c + q) * H + k) : "memory");
        v[q] = fmaf(__ldg(r + k), x, v[q]);
      }
    }
    send16(dst, bar, v);
  }
}

// ITEMS: 16-byte words of h a thread brings in per step, at most.
template <int ITEMS>
__global__ void __launch_bounds__(THREADS, 1) lstm_cluster_kernel(const ClusterArgs a) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ ClusterShared sh;
  unsigned char* h_hi = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int kblk = (a.kc + 31) / 32;                       // 32-wide K blocks of the h operand
  const uint32_t blk_bytes = (uint32_t)a.n * 128u;
  const uint32_t lo_off = (uint32_t)kblk * blk_bytes;
  // partial sums received: [parity][source CTA][4 batch rows][gate][unit][batch row], so that the lanes of a warp
  // (consecutive gate rows) write consecutive 16-byte words of their destination
  float* recv = reinterpret_cast<float*>(h_hi + 2 * lo_off);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H;
  const int rank = (int)(blockIdx.x % CS), cluster = (int)(blockIdx.x / CS);
  const int group = cluster / a.blocks, block = cluster - group * a.blocks;
  const int b0 = a.b0 + group * a.per;                     // first batch row of this group
  const int nb = min(a.per, a.b0 + a.nb - b0);
  const int u0 = block * UNITS;                            // first unit of this cluster
  const int k0 = rank * a.kc, klen = max(0, min(a.kc, H - k0));

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.mma_bar)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.recv_bar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.recv_bar[1])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sh.abort = sh.plain_r = sh.plain_h = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // rows of h past the batch and columns past the slice stay zero for the whole sequence
  for (uint32_t i = (uint32_t)tid * 16u; i < 2u * lo_off; i += THREADS * 16u)
    *reinterpret_cast<float4*>(h_hi + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem_base;
  const uint32_t tmem_a = tmem + (uint32_t)D_COLS;
  if (warp < 4) {
    // gate row r of the cluster = gate r % 4 of unit r / 4; this thread's row of R, slice k0 .. k0 + kc
    const int r = tid, unit = u0 + r / 4;
    const float* src = a.R + ((size_t)(r & 3) * H + unit) * H + k0;
    const uint32_t dst = tmem_a + ((uint32_t)(warp * 32) << 16);
    bool plain = false;
    for (int c = 0; c < a.kc; c += 8) {
      float hi[8], lo[8];
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (unit < H && c + j < klen) v = __ldg(reinterpret_cast<const float4*>(src + c + j));
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++) {
          hi[j + q] = high_part(e[q]);
          lo[j + q] = e[q] - hi[j + q];
          plain |= not_finite(hi[j + q]);
        }
      }
      tmem_st8(dst + (uint32_t)c, hi);
      tmem_st8(dst + (uint32_t)(a.kc + c), lo);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    if (plain) sh.plain_r = 1;
  }
  // Pairs (unit, batch row) this thread finishes: consecutive threads are consecutive units of one row, so that a
  // row's units leave in one store and arrive as the 16-byte words its readers ask for.
  float c_reg[PAIRS], h_reg[PAIRS], bsum[PAIRS][4];
  const float* p_src[PAIRS];        // projected inputs of the next step
  float* y_dst[PAIRS];              // h of the next step
  const float* sum_src[PAIRS];      // this pair's first partial sum in `recv`
  bool live[PAIRS];
#pragma unroll
  for (int p = 0; p < PAIRS; p++) {
    const int i = tid + p * THREADS, ul = i % UPC, bl = i / UPC, u = u0 + rank * UPC + ul, b = b0 + bl;
    live[p] = bl < nb && u < H;
    c_reg[p] = h_reg[p] = 0.f;
#pragma unroll
    for (int g = 0; g < 4; g++) bsum[p][g] = 0.f;
    p_src[p] = a.P + (size_t)b * 4 * H + u;
    y_dst[p] = a.Y + (size_t)b * H + u;
    sum_src[p] = recv + ((bl >> 2) * ROWS + ul) * 4 + (bl & 3);
    if (live[p]) {
      if (a.c0) c_reg[p] = a.c0[(size_t)b * H + u];
      if (a.bias) {
#pragma unroll
        for (int g = 0; g < 4; g++) bsum[p][g] = a.bias[g * H + u] + a.bias[(4 + g) * H + u];
      }
    }
  }
  // words of h this thread brings in: where they are in a step's [B, H] and in the swizzled operand
  const int chunks = klen / 4;                             // 16-byte words of a row of the slice
  const int items = nb * chunks;
  int h_src[ITEMS];
  uint32_t h_dst[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const int i = tid + j * THREADS;
    h_src[j] = 0;
    h_dst[j] = 0;
    if (i < items) {
      const uint32_t row = (uint32_t)(i / chunks), ch = (uint32_t)(i % chunks);
      h_src[j] = (int)row * H + (int)ch * 4;
      h_dst[j] = (ch >> 3) * blk_bytes + row * 128u + (((ch & 7u) ^ (row & 7u)) << 4);
      if (a.h0) {   // (later h are products of a sigmoid and a tanh)
        const float4 e = *reinterpret_cast<const float4*>(a.h0 + (size_t)b0 * H + k0 + h_src[j]);
        if (not_finite(high_part(e.x)) || not_finite(high_part(e.y)) || not_finite(high_part(e.z)) || not_finite(high_part(e.w)))
          sh.plain_h = 1;
      }
    }
  }
  const uint32_t step_bytes = 128u * (uint32_t)a.n * 4u;   // all rows this CTA finishes, from every CTA of the cluster
  if (tid == 0) {
    for (int q = 0; q < 2; q++)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sh.recv_bar[q])),
                   "r"(step_bytes)
                   : "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_barrier();                                       // barriers of every CTA are ready for the others' bytes
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const bool plain_r = sh.plain_r != 0, plain_h = sh.plain_h != 0;
  const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(a.n >> 3) << 17) | ((128u >> 4) << 24);
  const uint64_t desc0 = make_smem_desc(smem_u32(h_hi));
  // where this thread's accumulator columns go: row r of the tile is finished by CTA r / ROWS of the cluster
  const int my_row = (warp & 3) * 32 + lane, half = warp >> 2, cols = a.n / 2;
  const uint32_t peer = (uint32_t)(my_row / ROWS);
  const int dest_row = my_row % ROWS, slot = (dest_row & 3) * UPC + dest_row / 4;
  const uint32_t parity_bytes = 128u * (uint32_t)a.n * 4u;
  const uint32_t recv_peer =
      map_to(smem_u32(recv) + (uint32_t)((rank * a.n / 4 + half * cols / 4) * ROWS + slot) * 16u, peer);
  const uint32_t bar_peer[2] = {map_to(smem_u32(&sh.recv_bar[0]), peer), map_to(smem_u32(&sh.recv_bar[1]), peer)};
  const uint32_t d_src = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * cols);

  for (int t = 0; t < a.T; t++) {
    // h_{t-1}, this CTA's columns
    const float* hsrc = t > 0 ? a.Y + (size_t)(t - 1) * a.B * H : a.h0;
    bool ok = true;
    uint4 v[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) v[j] = make_uint4(0, 0, 0, 0);
    if (hsrc) {
      hsrc += (size_t)b0 * H + k0;
#pragma unroll
      for (int j = 0; j < ITEMS; j++)
        if (tid + j * THREADS < items) v[j] = ld_relaxed(hsrc + h_src[j]);
    }
    // projected inputs of this step: asked for while the first look at h is on its way
    float pin[PAIRS][4];
#pragma unroll
    for (int p = 0; p < PAIRS; p++) {
      if (live[p]) {
#pragma unroll
        for (int g = 0; g < 4; g++) pin[p][g] = __ldg(p_src[p] + g * H);
        p_src[p] += (size_t)a.B * 4 * H;
      }
    }
    if (hsrc) {
      if (t > 0) {
        unsigned long long since = 0;
        for (int tries = 0;; tries++) {
          bool missing = false;
#pragma unroll
          for (int j = 0; j < ITEMS; j++)
            if (is_empty(v[j])) {
              v[j] = ld_relaxed(hsrc + h_src[j]);
              missing = true;
            }
          if (!missing) break;
          if ((tries & 1023) == 1023) {
            if (since == 0) since = global_ns();
            if (global_ns() - since > WAIT_NS) {
              atomicCAS(a.status, 0, 91);
              ok = false;
              break;
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < ITEMS; j++) {
        if (tid + j * THREADS < items) {
          const float e[4] = {__uint_as_float(v[j].x), __uint_as_float(v[j].y), __uint_as_float(v[j].z),
                              __uint_as_float(v[j].w)};
          float hi[4], lo[4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            hi[q] = high_part(e[q]);
            lo[q] = e[q] - hi[q];
          }
          *reinterpret_cast<float4*>(h_hi + h_dst[j]) = make_float4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<float4*>(h_hi + h_dst[j] + lo_off) = make_float4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
    }
    if (!ok) sh.abort = 1;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (sh.abort) break;
    if (warp == 0) {
      if (elect_one()) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t lo_step = lo_off >> 4, blk_step = blk_bytes >> 4;
        uint32_t dh = (uint32_t)desc0, ah = tmem_a, al = tmem_a + (uint32_t)a.kc;   // (the low word holds the address)
        const uint32_t top = (uint32_t)(desc0 >> 32);
        umma_step<true>(tmem, ah, al, dh, dh + lo_step, top, idesc);
        const int steps = a.kc / 8;
#pragma unroll
        for (int k = 1; k < 4; k++)
          if (k < steps) umma_step<false>(tmem, ah + k * 8, al + k * 8, dh + k * 2, dh + lo_step + k * 2, top, idesc);
        for (int k0 = 4; k0 < steps; k0 += 4) {
          dh += blk_step;
          ah += 32u;
          al += 32u;
#pragma unroll
          for (int k = 0; k < 4; k++)
            if (k0 + k < steps)
              umma_step<false>(tmem, ah + k * 8, al + k * 8, dh + k * 2, dh + lo_step + k * 2, top, idesc);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&sh.mma_bar))
                     : "memory");
      }
      __syncwarp();   // the other lanes would take turns with the issuing one while they poll
    }
    ok = mbar_wait(smem_u32(&sh.mma_bar), (uint32_t)(t & 1), a.status, 92);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t dst = recv_peer + (t & 1 ? parity_bytes : 0u);
      const uint32_t bar = bar_peer[t & 1];
      const bool plain = plain_r || (t == 0 && plain_h);
      if (plain) send_plain_sums(a.R, hsrc, H, nb, half * cols, cols, u0, my_row, k0, klen, dst, ROWS * 16u, bar);
      for (int c = 0; c < cols && !plain; c += 16) {
        float v[16];
        tmem_ld8(d_src + (uint32_t)c, v);
        if (c + 8 < cols) tmem_ld8(d_src + (uint32_t)(c + 8), v + 8);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 16; q += 4) {
          if (c + q < cols) send16(dst, bar, v + q);
          dst += ROWS * 16u;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      ok = mbar_wait(smem_u32(&sh.recv_bar[t & 1]), (uint32_t)((t >> 1) & 1), a.status, 93);
    }
    if (ok) {
#pragma unroll
      for (int p = 0; p < PAIRS; p++) {
        if (live[p]) {
          const float* s = sum_src[p] + (t & 1 ? 128 * a.n : 0);
          float part[CS][4];
#pragma unroll
          for (int q = 0; q < CS; q++)
#pragma unroll
            for (int g = 0; g < 4; g++) part[q][g] = s[q * (ROWS * a.n) + g * (UPC * 4)];
          float g4[4];
#pragma unroll
          for (int g = 0; g < 4; g++) {
            g4[g] = pin[p][g] + bsum[p][g];
#pragma unroll
            for (int q = 0; q < CS; q++) g4[g] += part[q][g];
          }
          const float it = sigmoid_ref(g4[0]), ot = sigmoid_ref(g4[1]), ft = sigmoid_ref(g4[2]), ct = tanhf(g4[3]);
          c_reg[p] = ft * c_reg[p] + it * ct;
          h_reg[p] = ot * tanhf(c_reg[p]);
          asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(y_dst[p]), "f"(h_reg[p]) : "memory");
          y_dst[p] += (size_t)a.B * H;
        }
      }
    } else {
      sh.abort = 1;
    }
    // (this barrier's next bytes are those of step t + 2, which no CTA sends before all have sent step t + 1)
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sh.recv_bar[t & 1])),
                   "r"(step_bytes)
                   : "memory");
  }
#pragma unroll
  for (int p = 0; p < PAIRS; p++) {
    if (live[p]) {
      const int i = tid + p * THREADS, u = u0 + rank * UPC + i % UPC, b = b0 + i / UPC;
      a.Yh[(size_t)b * H + u] = h_reg[p];
      a.Yc[(size_t)b * H + u] = c_reg[p];
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_barrier();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

typedef void (*Kernel)(const ClusterArgs);

// by the words of h per thread of a launch with n batch rows and a K slice of kc
Kernel kernel_of(int n, int kc) { return n * (kc / 4) <= 4 * THREADS ? lstm_cluster_kernel<4> : lstm_cluster_kernel<12>; }

size_t smem_of(int n, int kc) { return (size_t)n * ((kc + 31) / 32 * 256 + 2 * 128 * 4) + 1024; }

void fill_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int grid, size_t smem, cudaStream_t stream) {
  *cfg = {};
  cfg->gridDim = dim3((unsigned)grid);
  cfg->blockDim = dim3(THREADS);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 2;
}

// Clusters whose CTAs have `smem` bytes each that can be resident at once (asked once per device and shape).
int max_clusters(wdc_context* ctx, Kernel kernel, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<std::pair<int, Kernel>, size_t>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(std::make_pair(ctx->device, kernel), smem);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  fill_config(&cfg, attr, CS, smem, nullptr);
  cfg.numAttrs = 1;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known[key] = n;
  return n;
}

struct Plan {
  Kernel kernel = nullptr;
  int kc = 0, per = 0, n = 0;
  int fit = 0;            // groups of batch rows (each on `blocks` clusters) that are resident at once
  size_t smem = 0;
};

Plan plan_of(wdc_context* ctx, int64_t Bt, int64_t H, int blocks) {
  Plan p;
  p.kc = (int)((ceil_div64(H, CS) + 7) / 8 * 8);
  // batch rows per group: as few as spread the batch over the clusters that fit, at most what shared memory, the
  // threads' words of h and their (unit, row) pairs allow
  int most = PAIRS * THREADS / UPC < D_COLS ? PAIRS * THREADS / UPC : D_COLS;
  while (most > 16 && (smem_of(most, p.kc) > (size_t)MAX_SMEM || most * (p.kc / 4) > MAX_ITEMS * THREADS)) most -= 16;
  if (smem_of(most, p.kc) > (size_t)MAX_SMEM) return Plan();
  if (most > Bt) most = (int)Bt;
  const int most_n = (most + 15) / 16 * 16;
  p.fit = max_clusters(ctx, kernel_of(most_n, p.kc), smem_of(most_n, p.kc)) / blocks;
  if (!p.fit) return Plan();
  int groups = (int)ceil_div64(Bt, 16);        // an MMA has at least 16 columns
  if (groups > p.fit) groups = p.fit;
  p.per = (int)ceil_div64(Bt, groups);
  if (p.per > most) {                          // several launches: equal shares
    const int64_t launches = ceil_div64(Bt, (int64_t)most * p.fit);
    p.per = (int)ceil_div64(Bt, launches * p.fit);
  }
  p.n = (p.per + 15) / 16 * 16;
  p.kernel = kernel_of(p.n, p.kc);
  p.smem = smem_of(p.n, p.kc);
  if (max_clusters(ctx, p.kernel, p.smem) / blocks < p.fit) return Plan();
  return p;
}

}  // namespace

// Runs the recurrence on the projected input P.  WDC_ERR_UNSUPPORTED: shape outside the kernel's range, or not all
// clusters would be resident (nothing has been written but Y's filling); any other non-zero status is an error.
int wdc_lstm_cluster(wdc_context* ctx, const float* P, const float* R, const float* bias, const float* h0,
                     const float* c0, float* Y, float* Yh, float* Yc, int64_t T, int64_t Bt, int64_t H) {
  // One to three steps do not pay for filling Y and bringing R into tensor memory, and below 32 units most rows of the
  // MMA would be empty: the other paths keep those.
  if (T < 4 || H < UNITS) return WDC_ERR_UNSUPPORTED;
  if (T > (1 << 24) || Bt > (1 << 20) || H % 4 != 0 || H > CS * KC_MAX) return WDC_ERR_UNSUPPORTED;
  if ((((uintptr_t)R | (uintptr_t)Y | (uintptr_t)h0) & 15) != 0) return WDC_ERR_UNSUPPORTED;
  ClusterArgs a = {P, R, bias, h0, c0, Y, Yh, Yc, ctx->status_word, (int)T, (int)Bt, (int)H};
  a.blocks = (int)((H + UNITS - 1) / UNITS);
  const Plan p = plan_of(ctx, Bt, H, a.blocks);
  if (!p.fit) return WDC_ERR_UNSUPPORTED;
  a.per = p.per;
  a.n = p.n;
  a.kc = p.kc;
  WDC_CUDA(ctx, cudaMemsetAsync(Y, 0xff, (size_t)(T * Bt * H) * 4, ctx->stream));
  const int64_t share = (int64_t)p.per * p.fit;
  for (int64_t b0 = 0; b0 < Bt; b0 += share) {
    a.b0 = (int)b0;
    a.nb = (int)(Bt - b0 < share ? Bt - b0 : share);
    const int groups = (a.nb + a.per - 1) / a.per;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    fill_config(&cfg, attr, groups * a.blocks * CS, p.smem, ctx->stream);
    cudaError_t e = cudaLaunchKernelEx(&cfg, p.kernel, (const ClusterArgs)a);
    if (e != cudaSuccess) {
      cudaGetLastError();
      if (b0 == 0) return WDC_ERR_UNSUPPORTED;
      return wdc_check_cuda(ctx, e, "lstm_cluster_kernel");
    }
    ctx->n_tc_launch++;
    const int s = wdc_check_launch(ctx, "lstm_cluster_kernel");
    if (s != WDC_OK) return s;
  }
  return WDC_OK;
}
