// Products of two activations on the 5th-generation tensor cores (tcgen05, sm_100a): batched MatMul and any Gemm whose
// operands cannot be prepared beforehand (ragged K, any strides).
//
//   Y[b, m, n] = alpha * sum_k A[b, m, k] B[b, k, n] + beta * C[m, n]
//
// conv_tc.cu wants B split and laid out once per weight; here both operands are new at every call, so they are split
// on their way into shared memory and nothing is written to HBM in between.  One CTA per 128 x TN tile of the output:
//   * 256 threads load a K block (32 wide) of A and B from global memory into registers one block ahead, in whichever
//     of three access patterns is coalesced for the operand's strides, and write it to shared memory as the K-major
//     128B-swizzled operand twice: the value rounded to TF32 and the rest;
//   * one thread issues lo*hi + hi*lo + hi*hi (3xTF32) as 12 tcgen05.mma of M 128 x N TN x K 8, A and B both from
//     shared memory, into TMEM; the two stages let the loads and the split of a block overlap the MMAs before it;
//   * the TMEM accumulator holds at most 4 K blocks (the tensor core truncates when it aligns addends); segments are
//     added in fp32 registers, one segment behind the MMAs;
//   * the result leaves through shared memory, so that every store instruction writes consecutive columns.
// What bounds it at [8, 850, 32] x [8, 32, 850] is writing 23 MB.  An infinite or NaN operand would meet low parts of
// either sign or zero; a tile that contains one is recomputed with plain fp32 FMAs, which keeps IEEE results.
// Waits are bounded (2 s, status word) like everywhere.
#include <cuda.h>

#include "common.cuh"

namespace {

constexpr int TM = 128;              // rows of a tile = TMEM lanes
constexpr int KB = 32;               // K block: one 128-byte swizzle row
constexpr int SEG = 4;               // K blocks per TMEM segment
constexpr int THREADS = 256;
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;

struct DirectArgs {
  const float* A;
  const float* B;
  const float* C;                    // null: no addend
  float* Y;
  int64_t sab, sa_row, sa_k, sbb, sb_row, sb_k, sc0, sc1;   // "row" of B: a column of the product
  int m, n, k;
  int mode_a, mode_b;                // LOAD_*
  float alpha, beta;
  int relu;
  int* status;
};

enum { LOAD_VEC4 = 0, LOAD_K = 1, LOAD_ROW = 2 };

struct DirectShared {
  unsigned long long bar[2];         // a stage's MMAs have completed
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

// Registers of a thread's share of one K block of an operand with ROWS rows: ROWS / 8 floats.
//   LOAD_VEC4: K contiguous and 16-byte aligned: 8 threads x 16 bytes per row
//   LOAD_K:    lanes along K (any strides; coalesced when K is contiguous)
//   LOAD_ROW:  lanes along the rows (contiguous rows, e.g. B stored [k][n]); a thread holds 4 consecutive k of a row
template <int ROWS>
__device__ __forceinline__ void load_block(float* v, const float* base, int64_t s_row, int64_t s_k, int rows, int k0,
                                           int klen, int mode) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int i = 0; i < ROWS / 8; i++) v[i] = 0.f;
  if (mode == LOAD_VEC4) {
    const int k = k0 + (tid & 7) * 4;
    const float* p = base + (int64_t)(tid >> 3) * s_row + k;
    if (k < klen) {
#pragma unroll
      for (int i = 0; i < ROWS / 32; i++) {
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
      for (int i = 0; i < ROWS / 8; i++) {
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
        for (int i = 0; i < ROWS / 32; i++)
          if (lane + 32 * i < rows) v[4 * i + t] = pdl_ld(p + 32 * i);
      }
      p += s_k;
    }
  }
}

// Writes the registers of load_block as the swizzled operand (high parts) and, `lo_off` bytes behind, its low parts.
template <int ROWS>
__device__ __forceinline__ bool store_block(const float* v, unsigned char* hi, uint32_t lo_off, int mode) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float h[ROWS / 8];
  bool bad = false;
#pragma unroll
  for (int i = 0; i < ROWS / 8; i++) {
    h[i] = high_part(v[i]);
    bad |= not_finite(h[i]);
  }
  if (mode == LOAD_K) {
#pragma unroll
    for (int i = 0; i < ROWS / 8; i++) {
      const uint32_t row = (uint32_t)(warp + 8 * i);
      const uint32_t off = row * 128u + ((((uint32_t)lane >> 2) ^ (row & 7u)) << 4) + ((uint32_t)lane & 3u) * 4u;
      *reinterpret_cast<float*>(hi + off) = h[i];
      *reinterpret_cast<float*>(hi + off + lo_off) = v[i] - h[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < ROWS / 32; i++) {
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

// TN: tile width.  kLong: more than one TMEM segment (running sums live in registers).
template <int TN, bool kLong>
__global__ void __launch_bounds__(THREADS, kLong && TN == 128 ? 1 : 2) gemm_tc_direct_kernel(const DirectArgs a) {
  constexpr int A_BYTES = TM * 128, B_BYTES = TN * 128, STAGE = 2 * A_BYTES + 2 * B_BYTES;
  constexpr int COLS = TN / 2;                         // accumulator columns of a warp
  constexpr int NBUF = kLong ? 2 : 1;
  constexpr int TMEM_COLS = NBUF * TN < 32 ? 32 : NBUF * TN;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* stages = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ DirectShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * TN, m0 = blockIdx.y * TM;
  const int rows_a = a.m - m0 < TM ? a.m - m0 : TM, rows_b = a.n - n0 < TN ? a.n - n0 : TN;
  const int kblocks = (a.k + KB - 1) / KB;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.bar[0])));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.bar[1])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sh.ok = 1;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  pdl_grid_wait();
  const float* C = pdl_after(a.C);
  const float* A = pdl_after(a.A) + blockIdx.z * a.sab + (int64_t)m0 * a.sa_row;
  const float* B = pdl_after(a.B) + blockIdx.z * a.sbb + (int64_t)n0 * a.sb_row;
  float va[TM / 8], vb[TN / 8];
  load_block<TM>(va, A, a.sa_row, a.sa_k, rows_a, 0, a.k, a.mode_a);
  load_block<TN>(vb, B, a.sb_row, a.sb_k, rows_b, 0, a.k, a.mode_b);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_let_next_start();   // not before this CTA has its tensor memory: a CTA of the next grid might take it and wait for this one
  const uint32_t tmem_base = sh.tmem_base;
  // D = f32, A = B = tf32, both K-major, M = 128, N = TN
  const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);

  float acc[COLS];
#pragma unroll
  for (int c = 0; c < COLS; c++) acc[c] = 0.f;
  const uint32_t my_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * COLS);
  auto drain = [&](int buf) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
      float t[16];
      tmem_ld16(my_lane + (uint32_t)(buf * TN + c), t);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 16; j++) acc[c + j] += t[j];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  };

  bool bad = false, ok = true;
  for (int kb = 0; kb < kblocks; kb++) {
    const int st = kb & 1;
    unsigned char* sb = stages + st * STAGE;
    // the stage's previous MMAs (two blocks ago) have read it
    if (kb >= 2) ok = mbar_wait(&sh.bar[st], (uint32_t)(((kb >> 1) - 1) & 1), a.status, 81);
    bad |= store_block<TM>(va, sb, A_BYTES, a.mode_a);
    bad |= store_block<TN>(vb, sb + 2 * A_BYTES, B_BYTES, a.mode_b);
    if (!ok) sh.ok = 0;
    if (kb + 1 < kblocks) {
      load_block<TM>(va, A, a.sa_row, a.sa_k, rows_a, (kb + 1) * KB, a.k, a.mode_a);
      load_block<TN>(vb, B, a.sb_row, a.sb_k, rows_b, (kb + 1) * KB, a.k, a.mode_b);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (!sh.ok) break;            // uniform: written before the barrier above
    const int seg = kb / SEG, buf = kLong ? seg & 1 : 0;
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t s0 = smem_u32(sb);
      const uint64_t ah = make_smem_desc(s0), al = make_smem_desc(s0 + A_BYTES);
      const uint64_t bh = make_smem_desc(s0 + 2 * A_BYTES), bl = make_smem_desc(s0 + 2 * A_BYTES + B_BYTES);
      const uint32_t d = tmem_base + (uint32_t)(buf * TN);
#pragma unroll
      for (int k8 = 0; k8 < KB / 8; k8++) {
        const uint64_t adv = (uint64_t)(k8 * 2);
        umma_tf32_ss(d, al + adv, bh + adv, idesc, ((kLong ? kb % SEG : kb) | k8) ? 1u : 0u);
        umma_tf32_ss(d, ah + adv, bl + adv, idesc, 1u);
        umma_tf32_ss(d, ah + adv, bh + adv, idesc, 1u);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&sh.bar[st]))
                   : "memory");
    }
    // The segment before this one: its last block's MMAs completed when this segment's second block found its stage
    // free.  (Its TMEM buffer is written again only by the segment after this one, behind the barriers in between.)
    if (kLong && kb % SEG == 1 && seg > 0) drain((seg - 1) & 1);
  }
  if (ok && sh.ok) {
    // all MMAs complete in order: the last commit stands for all of them
    ok = mbar_wait(&sh.bar[(kblocks - 1) & 1], (uint32_t)(((kblocks - 1) >> 1) & 1), a.status, 82);
    const int last = (kblocks - 1) / SEG;
    if (ok && kLong) {
      // a last segment of one block has not passed the in-loop drain of the segment before it
      if (last > 0 && (kblocks - 1) % SEG == 0) drain((last - 1) & 1);
      drain(last & 1);
    } else if (ok) {
      drain(0);
    }
  }
  const int any_bad = __syncthreads_or(bad ? 1 : 0);
  const bool done = ok && sh.ok;
  // the stages are free now: 32 x (COLS + 1) floats per warp to turn rows into consecutive columns
  float* stg = reinterpret_cast<float*>(stages) + warp * 32 * (COLS + 1);
  const int row0 = m0 + (warp & 3) * 32, col0 = n0 + (warp >> 2) * COLS;
  if (any_bad) {
    const int r = row0 + lane;
    for (int c = 0; c < COLS; c++) {
      float s = 0.f;
      if (r < a.m && col0 + c < a.n) {
        const float* pa = A + (int64_t)(r - m0) * a.sa_row;
        const float* pb = B + (int64_t)(col0 - n0 + c) * a.sb_row;
        for (int k = 0; k < a.k; k++) s = fmaf(pdl_ld(pa + (int64_t)k * a.sa_k), pdl_ld(pb + (int64_t)k * a.sb_k), s);
      }
      stg[lane * (COLS + 1) + c] = s;
    }
  } else {
#pragma unroll
    for (int c = 0; c < COLS; c++) stg[lane * (COLS + 1) + c] = acc[c];
  }
  __syncwarp();
  if (done) {
    float* Y = a.Y + (int64_t)blockIdx.z * a.m * a.n;
    for (int r = 0; r < 32 && row0 + r < a.m; r++) {
#pragma unroll
      for (int c = lane; c < COLS; c += 32) {
        if (col0 + c < a.n) {
          float v = stg[r * (COLS + 1) + c] * a.alpha;
          if (C) v += pdl_ld(C + (int64_t)(row0 + r) * a.sc0 + (int64_t)(col0 + c) * a.sc1) * a.beta;
          if (a.relu) v = v > 0.f ? v : (v == v ? 0.f : v);
          Y[(int64_t)(row0 + r) * a.n + col0 + c] = v;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
  }
}

template <int TN, bool kLong>
int launch(wdc_context* ctx, const DirectArgs& a, int batch) {
  constexpr int STAGE = 2 * TM * 128 + 2 * TN * 128;
  // a single K block needs one stage only: three CTAs per SM instead of one or two
  const int stages = a.k > KB ? 2 : 1;
  const int out = 8 * 32 * (TN / 2 + 1) * 4;
  const int smem = (stages * STAGE > out ? stages * STAGE : out) + 1024;
  static bool attr_set[64] = {};
  if (ctx->device < 0 || ctx->device >= 64) return WDC_ERR_UNSUPPORTED;
  if (!attr_set[ctx->device]) {
    if (cudaFuncSetAttribute(gemm_tc_direct_kernel<TN, kLong>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * STAGE + 1024) != cudaSuccess) {
      cudaGetLastError();
      return WDC_ERR_UNSUPPORTED;
    }
    attr_set[ctx->device] = true;
  }
  const dim3 grid((unsigned)((a.n + TN - 1) / TN), (unsigned)((a.m + TM - 1) / TM), (unsigned)batch);
  wdc_launch_pdl(ctx, gemm_tc_direct_kernel<TN, kLong>, dim3(grid), dim3(THREADS), smem, a);
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
