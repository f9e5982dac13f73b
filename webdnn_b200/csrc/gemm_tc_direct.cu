// Products of two activations on the 5th-generation tensor cores (tcgen05, sm_100a): batched MatMul and any Gemm whose
// operands cannot be prepared beforehand (ragged K, any strides).
//
//   Y[b, m, n] = alpha * sum_k A[b, m, k] B[b, k, n] + beta * C[m, n]
//
// conv_tc.cu wants B split and laid out once per weight; here both operands are new at every call, so they are split
// on their way into shared memory and nothing is written to HBM in between.  One CTA per 128 x TN tile of the output:
//   * groups of 256 threads load a K block (32 wide) of A and B from global memory into registers, the group's next one
//     ahead, in whichever of three access patterns is coalesced for the operand's strides, and write it to shared memory
//     as the K-major 128B-swizzled operand twice: the value rounded to TF32 and the rest;
//   * a warp of its own issues lo*hi + hi*lo + hi*hi (3xTF32) as 12 tcgen05.mma of M 128 x N TN x K 8, A and B both from
//     shared memory, into TMEM; loaders and issuer meet on a ring of stages, not at barriers of the whole CTA;
//   * the TMEM accumulator holds at most 4 K blocks (the tensor core truncates when it aligns addends); segments are
//     added in fp32 registers, one segment behind the MMAs;
//   * the result leaves through shared memory, in rows of consecutive 16- or 8-byte words where N and Y allow.
// Reductions of up to four K blocks are bound by a CTA's chain of latencies (load, split, MMA, output), so three or four CTAs
// share an SM.  Device time, before the ring and with it: [8, 850, 32] x [8, 32, 850] 20.3 -> 9.6 us (a call from the host takes
// 12), K = 64 31.6 -> 14.0, [64, 1024, 16] x [64, 16, 1024] 162 -> 74, [5, 1000, 32] x [5, 32, 77] 6.0 -> 4.3.  Longer ones: [3, 100, 1000]
// x [3, 1000, 77] 39 -> 23, [8, 850, 256] x [8, 256, 850] 57 -> 43, [64, 1024, 1024] x [64, 1024, 1024] 1450 -> 1250 (2600 cycles a K
// block, of which shared memory alone takes 1500: the MMAs read both operands there).
// An infinite or NaN operand would meet low parts of
// either sign or zero; a tile that contains one is recomputed with plain fp32 FMAs, which keeps IEEE results.
// Waits are bounded (2 s, status word) like everywhere.
#include <cuda.h>

#include "common.cuh"

namespace {

constexpr int TM = 128;              // rows of a tile = TMEM lanes
constexpr int KB = 32;               // K block: one 128-byte swizzle row
constexpr int SEG = 4;               // K blocks per TMEM segment
constexpr int MAX_STAGES = 4;
constexpr int SM_SMEM = 228 * 1024;
constexpr int GROUP = 256;           // threads that load a K block
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

struct DirectArgs {
  const float* A;
  const float* B;
  const float* C;                    // null: no addend
  float* Y;
  int64_t sab, sa_row, sa_k, sbb, sb_row, sb_k, sc0, sc1;   // "row" of B: a column of the product
  int m, n, k;
  int mode_a, mode_b;                // LOAD_*
  int stages;                        // K blocks in shared memory
  int vec;                           // consecutive columns of an aligned access of Y
  float alpha, beta;
  int relu;
  int* status;
};

enum { LOAD_VEC4 = 0, LOAD_K = 1, LOAD_ROW = 2 };

struct DirectShared {
  unsigned long long full[MAX_STAGES], empty[MAX_STAGES], seg_full[2], seg_empty[2];
  unsigned int tmem_base;
  int ok;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: false when the time limit passed (the status word then says so).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, int* status, int code) {
  for (int i = 0; i < 4096; i++)
    if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (;;) {
    for (int i = 0; i < 1024; i++)
      if (mbar_try_wait(bar, parity)) return true;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > WAIT_LIMIT_NS) {
      atomicCAS(status, 0, code);
      return false;
    }
  }
}
// shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void umma_tf32_ss(uint32_t tmem_c, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_c), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
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
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// x = high + low: the high part rounded to TF32 (11 bits), the low part exact before the tensor core cuts it, so that
// a product of the three terms kept is good to 2^-23
__device__ __forceinline__ float high_part(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }

// Registers of a thread's share of one K block of an operand with ROWS rows (a group of threads shares it):
//   LOAD_VEC4: K contiguous and 16-byte aligned: 8 threads x 16 bytes per row
//   LOAD_K:    lanes along K (any strides; coalesced when K is contiguous)
//   LOAD_ROW:  lanes along the rows (contiguous rows, e.g. B stored [k][n]); a thread holds 4 consecutive k of a row
template <int ROWS>
struct Share {
  static_assert(ROWS * 8 % GROUP == 0, "every thread has a share");
  static constexpr int CELLS = ROWS * 8 / GROUP;                   // groups of four floats
  static constexpr int N = 4 * CELLS;
};
template <int ROWS>
__device__ __forceinline__ void load_block(float* v, const float* base, int64_t s_row, int64_t s_k, int rows, int k0,
                                           int klen, int mode) {
  using S = Share<ROWS>;
  const int tid = threadIdx.x % GROUP, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int i = 0; i < S::N; i++) v[i] = 0.f;
  if (mode == LOAD_VEC4) {
    const int k = k0 + (tid & 7) * 4;
    const float* p = base + (int64_t)(tid >> 3) * s_row + k;
    if (k < klen) {
#pragma unroll
      for (int i = 0; i < S::CELLS; i++) {
        if ((tid >> 3) + 32 * i < rows) {
          const float4 q = pdl_ld(reinterpret_cast<const float4*>(p));
          v[4 * i] = q.x; v[4 * i + 1] = q.y; v[4 * i + 2] = q.z; v[4 * i + 3] = q.w;
        }
        p += 32 * s_row;
      }
    }
  } else if (mode == LOAD_K) {
    const int k = k0 + lane;
    const float* p = base + (int64_t)warp * s_row + (int64_t)k * s_k;
    if (k < klen) {
#pragma unroll
      for (int i = 0; i < S::N; i++) {
        if (warp + 8 * i < rows) v[i] = pdl_ld(p);
        p += 8 * s_row;
      }
    }
  } else {
    const int k = k0 + warp * 4;
    const float* p = base + (int64_t)k * s_k + lane;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      if (k + t < klen) {
#pragma unroll
        for (int i = 0; i < S::CELLS; i++)
          if (lane + 32 * i < rows) v[4 * i + t] = pdl_ld(p + 32 * i);
      }
      p += s_k;
    }
  }
}

// Writes the registers of load_block as the swizzled operand (high parts) and, `lo_off` bytes behind, its low parts.
template <int ROWS>
__device__ __forceinline__ bool store_block(const float* v, unsigned char* hi, uint32_t lo_off, int mode) {
  using S = Share<ROWS>;
  const int tid = threadIdx.x % GROUP, warp = tid >> 5, lane = tid & 31;
  float h[S::N];
  bool bad = false;
#pragma unroll
  for (int i = 0; i < S::N; i++) {
    h[i] = high_part(v[i]);
    bad |= not_finite(h[i]);
  }
  if (mode == LOAD_K) {
#pragma unroll
    for (int i = 0; i < S::N; i++) {
      const uint32_t row = (uint32_t)(warp + 8 * i);
      const uint32_t off = row * 128u + ((((uint32_t)lane >> 2) ^ (row & 7u)) << 4) + ((uint32_t)lane & 3u) * 4u;
      *reinterpret_cast<float*>(hi + off) = h[i];
      *reinterpret_cast<float*>(hi + off + lo_off) = v[i] - h[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < S::CELLS; i++) {
      const uint32_t row = (uint32_t)((mode == LOAD_VEC4 ? tid >> 3 : lane) + 32 * i);
      const uint32_t chunk = (uint32_t)(mode == LOAD_VEC4 ? tid & 7 : warp);
      const uint32_t off = row * 128u + ((chunk ^ (row & 7u)) << 4);
      const float *q = v + 4 * i, *g = h + 4 * i;
      *reinterpret_cast<float4*>(hi + off) = make_float4(g[0], g[1], g[2], g[3]);
      *reinterpret_cast<float4*>(hi + off + lo_off) =
          make_float4(q[0] - g[0], q[1] - g[1], q[2] - g[2], q[3] - g[3]);
    }
  }
  return bad;
}

// A warp's 32 rows x COLS columns of sums, staged in shared memory, to Y: V consecutive columns per lane.  Several accesses of
// a lane at a time, and the questions for an addend and a Relu (EXTRA) outside: one by one, with a branch each, the loads
// from shared memory are a chain ([5, 1000, 32] x [5, 32, 77], 4-byte stores, 7.2 us and not 4.3).
template <int V, bool EXTRA, int COLS, int PITCH>
__device__ __forceinline__ void write_rows(const DirectArgs& a, const float* stg, float* Y, const float* C, int row0, int col0) {
  constexpr int LANES = COLS / V < 32 ? COLS / V : 32;             // of a row
  constexpr int ROWS = 32 / LANES;                                 // rows of an access
  constexpr int PER_ROW = COLS / (LANES * V), ITEMS = 32 / ROWS * PER_ROW, BATCH = V == 4 ? 4 : 8;
  static_assert(ITEMS % BATCH == 0, "whole batches");
  const int lane = threadIdx.x & 31, lr = lane / LANES, lc = lane % LANES * V;
  const int rows = a.m - row0, cols = a.n - col0 - lc;
  Y += (int64_t)(row0 + lr) * a.n + col0 + lc;
#pragma unroll 1
  for (int i0 = 0; i0 < ITEMS; i0 += BATCH) {
    float v[BATCH][V];
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const float* src = stg + (lr + (i0 + i) / PER_ROW * ROWS) * PITCH + lc + (i0 + i) % PER_ROW * (LANES * V);
      if (V == 4) *reinterpret_cast<float4*>(v[i]) = *reinterpret_cast<const float4*>(src);
      else if (V == 2) *reinterpret_cast<float2*>(v[i]) = *reinterpret_cast<const float2*>(src);
      else v[i][0] = src[0];
    }
#pragma unroll
    for (int i = 0; i < BATCH; i++) {
      const int r = (i0 + i) / PER_ROW * ROWS, c = (i0 + i) % PER_ROW * (LANES * V);
      if (lr + r >= rows || c >= cols) continue;
#pragma unroll
      for (int j = 0; j < V; j++) {
        v[i][j] *= a.alpha;
        if (EXTRA && C) v[i][j] += pdl_ld(C + (int64_t)(row0 + lr + r) * a.sc0 + (int64_t)(col0 + lc + c + j) * a.sc1) * a.beta;
        if (EXTRA && a.relu) v[i][j] = v[i][j] > 0.f ? v[i][j] : (v[i][j] == v[i][j] ? 0.f : v[i][j]);
      }
      float* dst = Y + (int64_t)r * a.n + c;
      if (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[i][0], v[i][1 % V], v[i][2 % V], v[i][3 % V]);
      else if (V == 2) *reinterpret_cast<float2*>(dst) = make_float2(v[i][0], v[i][1 % V]);
      else dst[0] = v[i][0];
    }
  }
}

// TN: tile width.  kLong: more than one TMEM segment (running sums live in registers).
template <int TN, bool kLong>
struct DirectLayout {
  static constexpr int A_BYTES = TM * 128, B_BYTES = TN * 128, STAGE = 2 * A_BYTES + 2 * B_BYTES;
  static constexpr int STAGES = TN == 128 ? 3 : 4;     // at most
  // Threads that load, split, add up and write (a warp more issues the MMAs).  A K block's way through a warp (wait,
  // split, write, proxy fence, arrive, ask for the next) takes 3000 cycles whatever the number of warps that share it, its
  // MMAs 800: where a CTA has the SM to itself, two groups of warps take alternate K blocks.
  static constexpr int GROUPS = kLong ? 2 : 1;
  static constexpr int LOADERS = GROUP * GROUPS, MMA_WARP = LOADERS / 32, THREADS = LOADERS + 32;
  static constexpr int CTAS = !kLong ? (TN == 32 ? 4 : 3) : 1;   // of an SM, at most
  static constexpr int COLS = TN * 128 / LOADERS < 16 ? 16 : TN * 128 / LOADERS;   // accumulator columns of a warp
  static constexpr int OUT_WARPS = TN / COLS * 4;      // warps that have some
  static constexpr int OUT_PITCH = COLS + 4;           // floats of a staged row: 16-byte cells, no bank conflicts
  static constexpr int OUT = OUT_WARPS * 32 * OUT_PITCH * 4;
};

template <int TN, bool kLong>
__global__ void __launch_bounds__(DirectLayout<TN, kLong>::THREADS, DirectLayout<TN, kLong>::CTAS) gemm_tc_direct_kernel(const DirectArgs a) {
  using L = DirectLayout<TN, kLong>;
  constexpr int COLS = L::COLS, MMA_WARP = L::MMA_WARP;
  constexpr int NBUF = kLong ? 2 : 1;
  constexpr int TMEM_COLS = NBUF * TN < 32 ? 32 : NBUF * TN;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ DirectShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * TN, m0 = blockIdx.y * TM;
  const int rows_a = a.m - m0 < TM ? a.m - m0 : TM, rows_b = a.n - n0 < TN ? a.n - n0 : TN;
  const int kblocks = (a.k + KB - 1) / KB, last_seg = (kblocks - 1) / SEG;

  if (tid < 2 * MAX_STAGES + 4) {
    unsigned long long* bar = tid < MAX_STAGES ? &sh.full[tid] : tid < 2 * MAX_STAGES ? &sh.empty[tid - MAX_STAGES]
                            : tid < 2 * MAX_STAGES + 2 ? &sh.seg_full[tid - 2 * MAX_STAGES] : &sh.seg_empty[tid - 2 * MAX_STAGES - 2];
    const int count = tid < MAX_STAGES || tid >= 2 * MAX_STAGES + 2 ? tid < MAX_STAGES ? GROUP / 32 : L::OUT_WARPS : 1;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid == 64) sh.ok = 1;
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  pdl_grid_wait();
  const float* C = pdl_after(a.C);
  const float* A = pdl_after(a.A) + blockIdx.z * a.sab + (int64_t)m0 * a.sa_row;
  const float* B = pdl_after(a.B) + blockIdx.z * a.sbb + (int64_t)n0 * a.sb_row;
  const int group = tid / GROUP;
  float va[Share<TM>::N], vb[Share<TN>::N];
  if (warp < MMA_WARP && group < kblocks) {
    load_block<TM>(va, A, a.sa_row, a.sa_k, rows_a, group * KB, a.k, a.mode_a);
    load_block<TN>(vb, B, a.sb_row, a.sb_k, rows_b, group * KB, a.k, a.mode_b);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_let_next_start();   // not before this CTA has its tensor memory: a CTA of the next grid might take it and wait for this one
  const uint32_t tmem_base = sh.tmem_base;

  float acc[kLong ? COLS : 1];
#pragma unroll
  for (int c = 0; c < (kLong ? COLS : 1); c++) acc[c] = 0.f;
  const uint32_t my_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * COLS);
  bool bad = false, ok = true;
  int drained = 0;
  auto drain = [&]() {   // the next segment's sums, behind those before it
    const int buf = drained & 1;
    ok = __all_sync(0xffffffffu, mbar_wait(&sh.seg_full[buf], (uint32_t)(drained >> 1) & 1u, a.status, 82));
    if (!ok) return;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int c = 0; c < (kLong ? COLS : 0); c += 16) {
      float t[16];
      tmem_ld16(my_lane + (uint32_t)(buf * TN + c), t);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 16; j++) acc[c + j] += t[j];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh.seg_empty[buf]);
    drained++;
  };

  if (warp < MMA_WARP) {
    int st = group;
    uint32_t par = 1;              // of the stage's release: the first round waits for nobody
    for (int kb = group; kb < kblocks; kb += L::GROUPS) {
      unsigned char* sb = stages + st * L::STAGE;
      // the stage's last MMAs have read it (MMAs complete in order, so the release before that is long past)
      if (kb >= a.stages) ok = __all_sync(0xffffffffu, mbar_wait(&sh.empty[st], par, a.status, 81));
      if (!ok) break;
      bad |= store_block<TM>(va, sb, L::A_BYTES, a.mode_a);
      bad |= store_block<TN>(vb, sb + 2 * L::A_BYTES, L::B_BYTES, a.mode_b);
      if (kb + L::GROUPS < kblocks) {
        load_block<TM>(va, A, a.sa_row, a.sa_k, rows_a, (kb + L::GROUPS) * KB, a.k, a.mode_a);
        load_block<TN>(vb, B, a.sb_row, a.sb_k, rows_b, (kb + L::GROUPS) * KB, a.k, a.mode_b);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.full[st]);
      st += L::GROUPS;
      if (st >= a.stages) { st -= a.stages; par ^= 1u; }
      // the segment before this block's, complete by now or soon; its buffer is wanted two blocks on
      if (kLong && kb % SEG == SEG - 2 + group && kb > SEG && warp < L::OUT_WARPS) {
        drain();
        if (!ok) break;
      }
    }
    while (kLong && ok && warp < L::OUT_WARPS && drained <= last_seg) drain();
    if (!kLong && ok) ok = mbar_wait(&sh.seg_full[0], 0, a.status, 82);
    if (!ok) sh.ok = 0;
  } else if (elect_one()) {
    // D = f32, A = B = tf32, both K-major, M = 128, N = TN
    constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
    const uint64_t desc0 = make_smem_desc(smem_u32(stages));
    int st = 0;
    uint32_t par = 0;
    for (int kb = 0; kb < kblocks && ok; kb++) {
      const int seg = kLong ? kb / SEG : 0, buf = seg & 1, in_seg = kLong ? kb % SEG : kb;
      if (kLong && in_seg == 0 && seg >= 2) ok = mbar_wait(&sh.seg_empty[buf], (uint32_t)((seg >> 1) - 1) & 1u, a.status, 83);
      ok = ok && mbar_wait(&sh.full[st], par, a.status, 84);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t ah = desc0 + (uint64_t)(st * (L::STAGE >> 4)), al = ah + (uint64_t)(L::A_BYTES >> 4);
      const uint64_t bh = al + (uint64_t)(L::A_BYTES >> 4), bl = bh + (uint64_t)(L::B_BYTES >> 4);
      const uint32_t d = tmem_base + (uint32_t)(buf * TN);
#pragma unroll
      for (int k8 = 0; k8 < KB / 8; k8++) {
        const uint64_t adv = (uint64_t)(k8 * 2);
        umma_tf32_ss(d, al + adv, bh + adv, idesc, (in_seg | k8) ? 1u : 0u);
        umma_tf32_ss(d, ah + adv, bl + adv, idesc, 1u);
        umma_tf32_ss(d, ah + adv, bh + adv, idesc, 1u);
      }
      if (kLong || kb + a.stages < kblocks) umma_commit(&sh.empty[st]);   // (nobody waits for the last ones)
      if (kb == kblocks - 1 || (kLong && in_seg == SEG - 1)) umma_commit(&sh.seg_full[buf]);
      if (++st == a.stages) { st = 0; par ^= 1u; }
    }
    if (!ok) sh.ok = 0;
  }
  const int any_bad = __syncthreads_or(bad ? 1 : 0);
  if (warp < L::OUT_WARPS && sh.ok) {
    // The stages are free now.  A warp turns its 32 rows into consecutive columns there; what it writes, it reads itself.
    float* stg = reinterpret_cast<float*>(stages) + warp * 32 * L::OUT_PITCH;
    const int row0 = m0 + (warp & 3) * 32, col0 = n0 + (warp >> 2) * COLS;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
      float t[16];
      if (kLong) {
#pragma unroll
        for (int j = 0; j < 16; j++) t[j] = acc[kLong ? c + j : 0];
      } else {
        tmem_ld16(my_lane + (uint32_t)c, t);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
#pragma unroll
      for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<float4*>(stg + lane * L::OUT_PITCH + c + j) = make_float4(t[j], t[j + 1], t[j + 2], t[j + 3]);
    }
    if (any_bad) {
      const int r = row0 + lane;
      for (int c = 0; c < COLS; c++) {
        float s = 0.f;
        if (r < a.m && col0 + c < a.n) {
          const float* pa = A + (int64_t)(r - m0) * a.sa_row;
          const float* pb = B + (int64_t)(col0 - n0 + c) * a.sb_row;
          for (int k = 0; k < a.k; k++) s = fmaf(pdl_ld(pa + (int64_t)k * a.sa_k), pdl_ld(pb + (int64_t)k * a.sb_k), s);
        }
        stg[lane * L::OUT_PITCH + c] = s;
      }
    }
    __syncwarp();
    float* Y = a.Y + (int64_t)blockIdx.z * a.m * a.n;
    if (C || a.relu) {
      if (a.vec == 4) write_rows<4, true, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
      else if (a.vec == 2) write_rows<2, true, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
      else write_rows<1, true, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
    } else {
      if (a.vec == 4) write_rows<4, false, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
      else if (a.vec == 2) write_rows<2, false, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
      else write_rows<1, false, COLS, L::OUT_PITCH>(a, stg, Y, C, row0, col0);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
  }
}

template <int TN, bool kLong>
int launch(wdc_context* ctx, DirectArgs a, int batch) {
  using L = DirectLayout<TN, kLong>;
  const dim3 grid((unsigned)((a.n + TN - 1) / TN), (unsigned)((a.m + TM - 1) / TM), (unsigned)batch);
  const int kblocks = (a.k + KB - 1) / KB;
  // Stages of short reductions: as many as leave room for all tiles at once ([16, 384, 128] x [16, 128, 384], 288 tiles: two
  // 11.0 us, one 15.4).  More tiles than that live on three or four CTAs per SM, one's output under the other's loads, with one
  // stage each (two at K = 64, [8, 850, 64] x [8, 64, 850]: one CTA an SM, 31.6 us and not 17.7).
  const int64_t tiles = (int64_t)grid.x * grid.y * grid.z;
  a.stages = kblocks < L::STAGES ? kblocks : L::STAGES;
  while (!kLong && a.stages > 1 && tiles > (int64_t)ctx->sm_count * (SM_SMEM / (a.stages * L::STAGE + 2048))) a.stages--;
  const int smem = (a.stages * L::STAGE > L::OUT ? a.stages * L::STAGE : L::OUT) + 1024;
  static bool attr_set[64] = {};
  if (ctx->device < 0 || ctx->device >= 64) return WDC_ERR_UNSUPPORTED;
  if (!attr_set[ctx->device]) {
    if (cudaFuncSetAttribute(gemm_tc_direct_kernel<TN, kLong>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             L::STAGES * L::STAGE + 1024) != cudaSuccess) {
      cudaGetLastError();
      return WDC_ERR_UNSUPPORTED;
    }
    attr_set[ctx->device] = true;
  }
  wdc_launch_pdl(ctx, gemm_tc_direct_kernel<TN, kLong>, dim3(grid), dim3(L::THREADS), smem, a);
  ctx->n_tc_launch++;
  return wdc_check_launch(ctx, "gemm_tc_direct_kernel");
}

template <int TN>
int launch_tn(wdc_context* ctx, const DirectArgs& a, int batch) {
  return a.k > SEG * KB ? launch<TN, true>(ctx, a, batch) : launch<TN, false>(ctx, a, batch);
}

}  // namespace

// WDC_ERR_UNSUPPORTED (nothing written): outside the kernel's index range.
int wdc_tc_gemm_direct(wdc_context* ctx, const wdc_gemm_desc* d, const float* A, const float* B, const float* C,
                       float* Y) {
  const int64_t limit = (1ll << 31) - 256;
  if (d->m >= limit || d->n >= limit || d->k >= limit || d->k < 1 || d->batch > 65535 || ceil_div64(d->m, TM) > 65535)
    return WDC_ERR_UNSUPPORTED;
  DirectArgs a = {};
  a.A = A; a.B = B; a.C = C; a.Y = Y;
  a.sab = d->sab; a.sa_row = d->sa0; a.sa_k = d->sa1;
  a.sbb = d->sbb; a.sb_row = d->sb1; a.sb_k = d->sb0;
  a.sc0 = d->sc0; a.sc1 = d->sc1;
  a.m = (int)d->m; a.n = (int)d->n; a.k = (int)d->k;
  a.vec = a.n % 4 == 0 && ((uintptr_t)Y & 15) == 0 ? 4 : a.n % 2 == 0 && ((uintptr_t)Y & 7) == 0 ? 2 : 1;
  a.alpha = d->alpha; a.beta = d->beta; a.relu = d->relu; a.status = ctx->status_word;
  auto mode = [&](const float* p, int64_t s_batch, int64_t s_row, int64_t s_k) {
    if (s_k == 1 && s_row % 4 == 0 && s_batch % 4 == 0 && a.k % 4 == 0 && ((uintptr_t)p & 15) == 0) return (int)LOAD_VEC4;
    return s_row == 1 && s_k != 1 ? (int)LOAD_ROW : (int)LOAD_K;
  };
  a.mode_a = mode(A, a.sab, a.sa_row, a.sa_k);
  a.mode_b = mode(B, a.sbb, a.sb_row, a.sb_k);
  // The widest tile that still gives every SM one (two, where two fit): wide tiles read A least often.
  const int64_t rows = ceil_div64(a.m, TM) * d->batch;
  if (a.n > 64 && rows * ceil_div64(a.n, 128) >= ctx->sm_count) return launch_tn<128>(ctx, a, (int)d->batch);
  if (a.n > 32 && rows * ceil_div64(a.n, 64) >= ctx->sm_count / 2) return launch_tn<64>(ctx, a, (int)d->batch);
  return launch_tn<32>(ctx, a, (int)d->batch);
}
