// ONNX LSTM recurrence with the whole of R inside one thread-block cluster.
//
// What bounds a recurrence is the chain of one step.  lstm_cluster.cu spreads R over the chip, so that h crosses from
// cluster to cluster through L2 (a store and a poll, 1850 cycles) and partial sums cross each cluster (1500 cycles).
// Here a batch row's recurrence never leaves its cluster, and there is one exchange a step:
//   * a CTA owns 32 hidden units (128 gate rows = the 128 lanes of an MMA) over the whole of K, a cluster the whole of R
//     (up to 16 CTAs, 512 units); the batch is dealt to the clusters that fit on the chip, which run independently;
//   * R fits because it is kept as two fp16 parts with a power of two per row (4 bytes an element, in tensor memory, the
//     last low parts in shared memory), where TF32 parts take 8.  h is in (-1, 1) and has a constant scale.  Two parts of
//     11 rounded bits carry 23 bits (TF32 parts, cut by the tensor core: 22), the low one with a scale of 2^13 of its own, so
//     that elements down to 2^-28 of a row's largest have 22 bits.  Of what is smaller in R they miss up to 2^-49 of the largest.
//     Where that can show, in a sum that is smaller than 2^24 times all of it, what is missing is added with fp32 FMAs, at the
//     price of the elements' way through L2; elsewhere it costs a comparison (a step of [64, 512] 2.39 us without
//     small elements, 2.49 with one unit's weights at 1e-12 of the others, 5.6 with 128 such units; always added they took 3.4
//     and 73).  Small elements of h0 stay out of the parts and are added.  h below 2^-29 is good to 2^-51 absolutely.  An fp16
//     MMA covers twice the K of a TF32 one in the same time: M 128 x N 16 x K 16 takes 9 cycles, N 32 takes 16;
//   * h goes to every CTA of the cluster as 16-byte words in the layout of the MMA's B operand (no swizzle: 8 batch rows x
//     8 units are 128 consecutive bytes), by st.async, whose mbarrier counts the bytes (a CTA takes in about 20 a clock:
//     16 KB of 8 rows x 512 units 800 cycles).  Barriers for each four sources, so that the first MMAs overlap the last
//     words, cost more than they gave (1.82 us a step for one, 1.82 to 1.74 for four at 16 rows, 1.49 to 1.63 at one);
//   * two buffers of h by the parity of the step: a CTA sends h_t after it has all of h_{t-1}, which every CTA sent after
//     its MMAs on h_{t-2}, the buffer's last reader, were complete.
// Measured, start of a step to the next with lstm_cluster.cu and here: 256 units, batch 1, 1.63 -> 0.85 us; [64, 512] 3.28 ->
// 2.39 us (of 4500 cycles the words on their way are 1500, 20 KB into every CTA, and the gates 940); 50 steps of [1, 256] with the
// projection 96 -> 58 us, 128 of [64, 512] 434 -> 343 us.
// Sums: hi*hi in one range of columns of an accumulator, hi*lo + lo*hi in another, added in fp32 after the last MMA.  The tensor
// core cuts every product off at the running sum's last bits, so a sum over K loses in proportion to K: the k steps go to four
// accumulators in turn.  Rms error of a sum of 480 (512) products against 64 bits: mixed signs 6.2e-7 (6.6e-7) in one accumulator,
// 2.1e-7 (2.1e-7) in four, 4.6e-7 (9.2e-7) by lstm_cluster.cu, whose CTAs sum slices of 60 (128); all of one sign 2.7e-6 (2.9e-6),
// 4.9e-7 (5.3e-7), 5.1e-7 (1.2e-6).  Their columns push low parts of R into shared memory, where an MMA takes 45 cycles more
// to read them: a step of [64, 512] 2.21 us in one accumulator, 2.30 in two, 2.50 in four; of [1, 256] 0.81, 0.80, 0.82.
// h0 may be anything: its rows have a scale each.  A row of R, or an h0, with an infinite element or NaN has none: all of it
// is left out of the parts.  Waits are bounded as in lstm_cluster.cu: on expiry a status word is set, the peers' waits expire in turn, and
// all CTAs of the cluster meet at the last barrier.
#include <cuda_fp16.h>
#include <math.h>

#include "common.cuh"

namespace {

constexpr int EPI_THREADS = 256;
constexpr int THREADS = EPI_THREADS + 32;   // warps 0-7: gates; warp 8: issues the MMAs
constexpr int UNITS = 32;                   // units of a CTA
constexpr int MAX_CS = 16;
constexpr int MAX_GROUPS = 4;               // 8-row groups of a cluster's batch rows
constexpr int QUARTERS = MAX_CS / 4;
constexpr int MAX_SMEM = 224 * 1024;
constexpr int MIN_SMEM = 116 * 1024;        // all of tensor memory is taken: one CTA per SM
constexpr float H_SCALE = 16384.f, H_UNSCALE = 1.f / 16384.f;
constexpr float LO_SCALE = 8192.f, LO_UNSCALE = 1.f / 8192.f;   // of low parts against high ones
constexpr float SMALL = 1.f / 32768.f;   // below that, scaled, the parts have fewer than 22 bits
constexpr unsigned long long WAIT_NS = 2000000000ull;

struct LocalArgs {
  const float* P;      // [T, B, 4H] input projection without bias
  const float* R;      // [4H, H]
  const float* bias;   // [8H] or null
  const float* h0;     // [B, H] or null
  const float* c0;
  float* Y;            // [T, B, H]
  float* Yh;
  float* Yc;
  int* status;
  int T, B, H;
  int cs;              // CTAs of a cluster: ceil(H / 32)
  int per;             // batch rows of a cluster
  unsigned int beyond;          // bytes of h waited for beyond those that come: 0 (the self-test: one word)
  unsigned long long wait_ns;   // limit of every wait (WAIT_NS; the self-test passes about a millisecond)
  int r_early;         // R is read before the grids in front have finished: a constant that nothing still running writes
};

struct LocalShared {
  unsigned long long mma_bar;
  unsigned long long full[2];
  unsigned int small_r[4][MAX_CS], small_h0[MAX_CS];   // units with small elements: of 32 rows of R, of h0; by source
  unsigned int tmem_base;
  float row_max[128];                 // later: of pack_row
  float h0_unscale[8 * MAX_GROUPS];   // negative: all of the row is left out of the parts
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
__device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, int* status, int code, unsigned long long limit_ns) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 256; i++)
      if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) {
      atomicCAS(status, 0, code);
      return false;
    }
  }
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const LocalArgs& a, int code) {
  for (int i = 0; i < 1024; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, a.status, code, a.wait_ns);
}
__device__ __forceinline__ void expect_bytes(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t map_to(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send16(uint32_t dst, uint32_t bar, const uint4& v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }
// Operand in shared memory, K-major without swizzle: 8 rows x 16 bytes are consecutive; `k_step` bytes between such
// blocks along K, `row_step` along the rows.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t k_step, uint32_t row_step) {
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)(k_step >> 4) << 16 | (uint64_t)(row_step >> 4) << 32 | (uint64_t)1 << 46;
}
// The descriptors as their halves: only the low one (the start address) changes from MMA to MMA.
__device__ __forceinline__ void mma_ts(uint32_t tmem_c, uint32_t tmem_a, uint32_t b_lo, uint32_t b_top, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 d;\n\t"
      "mov.b64 d, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n\t}" ::"r"(tmem_c),
      "r"(tmem_a), "r"(b_lo), "r"(b_top), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_ts_more(uint32_t tmem_c, uint32_t tmem_a, uint32_t b_lo, uint32_t b_top, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 d;\n\t"
      "mov.b64 d, {%2, %3};\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n\t}" ::"r"(tmem_c),
      "r"(tmem_a), "r"(b_lo), "r"(b_top), "r"(idesc)
      : "memory");
}
__device__ __forceinline__ void mma_ss_more(uint32_t tmem_c, uint32_t a_lo, uint32_t a_top, uint32_t b_lo, uint32_t b_top,
                                            uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 d, a;\n\t"
      "mov.b64 a, {%1, %2};\n\t"
      "mov.b64 d, {%3, %4};\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, d, %5, p;\n\t}" ::"r"(tmem_c),
      "r"(a_lo), "r"(a_top), "r"(b_lo), "r"(b_top), "r"(idesc)
      : "memory");
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
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
// The gates without branches, so that a thread's calls overlap (five tanhf in a row took 700 cycles of a step of 2400), and
// no further from float64 than the forms by tanhf, 0.5 tanhf(0.5 x) + 0.5 and tanhf(x), at any magnitude.  Largest errors over
// all floats in units of 2^-24, those forms' in brackets: the sigmoid's absolute one 0.54 [0.58] below 0.25, 0.68 [0.95] below 1,
// 1.29 [1.38] to 1.25, 1.05 [1.16] to 2, 0.9 [1.03] past it; tanh's relative one 1.23 [3.33] below 0.65, 2.9 [2.9] to 1, 1.7 [1.8] to 1.25,
// 0.86 [1.0] past 1.5.
// Around zero both are odd polynomials, fitted to equal ripple by Lawson's reweighted least squares (C. L. Lawson, 1961): the
// sigmoid's below 1 for its absolute error (0.03 * 2^-24 before rounding), tanh's below 0.7 for its relative one (0.02).  Past
// that 1 / (1 + e^x) is small and so is what it is wrong by: the sigmoid is that or 1 minus it, and tanh(x) = 1 - 2 / (1 + e^2x).
// e^x = 2^(x log2 e): the exponent's rounding costs (|x| log2 e) 2^-25, which tanh wins back as a factor 1 + l ln 2.
__device__ __forceinline__ float exp2_of(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float inverse(float x) {                // of 1 .. infinity
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sigmoid_of(float x) {
  const float m = fabsf(x), u = x * x;
  float q = 1.63452805e-05f;
  q = fmaf(q, u, -0.000206102079f);
  q = fmaf(q, u, 0.00208133925f);
  q = fmaf(q, u, -0.0208329856f);
  q = fmaf(q, u, 0.249999985f);
  const float tail = inverse(1.f + exp2_of(m * 1.44269504f));
  return m < 1.f ? fmaf(x, q, 0.5f) : x < 0.f ? tail : 1.f - tail;
}
__device__ __forceinline__ float tanh_of(float x) {
  const float m = fabsf(x), u = x * x;
  float q = 0.00189566764f;
  q = fmaf(q, u, -0.00788331125f);
  q = fmaf(q, u, 0.0215710606f);
  q = fmaf(q, u, -0.0539209545f);
  q = fmaf(q, u, 0.133329839f);
  q = fmaf(q, u, -0.333333254f);
  float y;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(2.f * m), "f"(80.f));
  const float h = y * 1.44269504f, l = fmaf(y, 1.92596299e-8f, fmaf(y, 1.44269504f, -h));
  const float e = exp2_of(h), tail = inverse(1.f + fmaf(e, l * 0.693147181f, e));
  return copysignf(m < 0.7f ? fmaf(m * u, q, m) : fmaf(-2.f, tail, 1.f), x);
}
// x = hi + lo / 2^13 in fp16 parts (|x| <= 2^14, so that |lo| <= 2^15): 23 bits, past 2^-15 at least 22, below that to 2^-37
__device__ __forceinline__ void split_half(float x, __half* hi, __half* lo) {
  *hi = __float2half_rn(x);
  *lo = __float2half_rn((x - __half2float(*hi)) * LO_SCALE);
}
// Elements that the parts would not hold to 22 bits: below a row's limit; a limit of NaN is for all of a row.
__device__ __forceinline__ bool is_small(float v, float limit) { return v != 0.f && !(fabsf(v) >= limit); }
__device__ __forceinline__ uint32_t nonzero_words(const unsigned int* words) {                // bit i: word i of MAX_CS
  uint32_t mask = 0;
#pragma unroll
  for (int i = 0; i < MAX_CS; i++) mask |= words[i] ? 1u << i : 0u;
  return mask;
}
// Power of two that brings the largest magnitude `m` of a row into [2^13, 2^14) (a row of zeros or denormals: the largest
// that leaves its inverse a normal number).
__device__ __forceinline__ int row_exponent(float m) {
  const int e = (int)(__float_as_uint(m) >> 23) - 127;
  return min(13 - e, 100);
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }   // -126 <= e <= 127
// A row's scale, and the limit of its small elements, by its largest magnitude: NaN where that is not finite.
__device__ __forceinline__ int scale_exponent(float m) { return not_finite(m) ? 0 : row_exponent(m); }   // -114 .. 100
// 2^24 times what the parts miss of a row, with the exponent of its largest magnitude in the last bits.  (One word for both: with 512
// bytes more in front of them the operands in shared memory start 1 KB later, and a step of [64, 512] takes 2.56 us, not 2.37.)
__device__ __forceinline__ float pack_row(float m, float error) {
  return __uint_as_float((__float_as_uint(error * 0x1p24f) & ~0xffu) | __float_as_uint(m) >> 23);
}
__device__ __forceinline__ float error_of(float packed) {          // rounded up; infinite for a row that is not finite
  const uint32_t bits = __float_as_uint(packed);
  return (bits & 0xffu) == 0xffu ? __uint_as_float(0x7f800000u) : bits >> 8 ? __uint_as_float(bits | 0xffu) : 0.f;
}
__device__ __forceinline__ float row_magnitude(float packed) { return __uint_as_float((__float_as_uint(packed) & 0xffu) << 23); }   // for limit_of
__device__ __forceinline__ float limit_of(float m) { return not_finite(m) ? __uint_as_float(0x7fffffffu) : pow2(-row_exponent(m)) * SMALL; }

// h of one buffer: [source CTA][zeros? hi groups, lo groups][4 blocks of 8 units][8 batch rows][8 units], fp16.
// An odd number of groups has a group of zeros in front: the MMA of the low parts of R has at least 16 columns and
// adds to the range of columns that hi*lo is summed in; the zeros stand for the 8 columns in front of that range.
// ACCS: accumulators that the k steps go to in turn.  TURNS: every other k step's low parts of R are in shared memory (where an
// MMA takes 64 cycles to read them, part of it behind the others), not those that tensor memory has no room for.
template <int NG, int ACCS, bool TURNS>
struct LocalLayout {
  static constexpr int ZERO = NG & 1;
  static constexpr int GROUP = 512;                               // bytes of a group: 8 rows x 32 units
  static constexpr int SRC = (ZERO + 2 * NG) * GROUP;
  static constexpr int BUF = MAX_CS * SRC;                        // (fixed, so that operand addresses are constants)
  static constexpr int ACC = 16 * NG;                             // columns: hi*hi, then the cross products
  static constexpr int D_COLS = ACC * ACCS;
  static constexpr int LO_ROWS = 8 * (NG + ZERO);                 // columns of the MMA of the low parts
  static constexpr int LO_COL0 = 8 * (NG - ZERO);
  static constexpr int STAGE = 8 * NG * 128;                      // the eight warps' words on their way out
  // k steps whose low parts of R are in tensor memory
  static __host__ __device__ constexpr int steps_lo(int cs) {
    return TURNS ? cs : (512 - D_COLS) / 8 - 2 * cs < 2 * cs ? (512 - D_COLS) / 8 - 2 * cs : 2 * cs;
  }
};

// The MMAs of four sources (two k steps each).  One block of straight-line code whose addresses are constant offsets from
// bases in registers: 13 cycles an MMA.  With addresses computed for each it takes 28 to 65, with a block of constants for
// every quarter and buffer behind a switch 25.
struct Issue {
  uint32_t t_d, t_hi, t_lo;    // tensor memory: accumulators, high and low parts of R from these sources' columns on
  uint32_t b, b_top;           // descriptor of their words
  uint32_t r, r_top;           // descriptor of the low parts of R in shared memory
};
template <int NG, int ACCS, bool TURNS, bool ALL>    // ALL: four sources, low parts in tensor memory
__device__ __forceinline__ void issue_sources(const Issue& o, int q, int n, int lo_in_tmem) {
  using L = LocalLayout<NG, ACCS, TURNS>;
  constexpr uint32_t ID_HI = (1u << 4) | ((uint32_t)(2 * NG) << 17) | ((128u >> 4) << 24);
  constexpr uint32_t ID_LO = (1u << 4) | ((uint32_t)(L::LO_ROWS >> 3) << 17) | ((128u >> 4) << 24);
#pragma unroll
  for (int d = 0; d < 4; d++) {
    if (ALL || d < n) {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int step = 2 * d + j;
        const uint32_t t_acc = o.t_d + (uint32_t)(step % ACCS * L::ACC);
        const uint32_t b = o.b + (uint32_t)((d * L::SRC + 256 * j) >> 4), b_hi = b + (uint32_t)(L::ZERO * L::GROUP >> 4);
        if (step < ACCS) mma_ts(t_acc, o.t_hi + (uint32_t)(8 * step), b_hi, o.b_top, ID_HI, q > 0 ? 1u : 0u);
        else mma_ts_more(t_acc, o.t_hi + (uint32_t)(8 * step), b_hi, o.b_top, ID_HI);
        // (with zeros in front: their 8 columns have just been written by the MMA above, like the others)
        if (TURNS && j == 1) mma_ss_more(t_acc + (uint32_t)L::LO_COL0, o.r + (uint32_t)(d * 256), o.r_top, b, o.b_top, ID_LO);
        else if (TURNS) mma_ts_more(t_acc + (uint32_t)L::LO_COL0, o.t_lo + (uint32_t)(8 * d), b, o.b_top, ID_LO);
        else if (ALL || step < lo_in_tmem) mma_ts_more(t_acc + (uint32_t)L::LO_COL0, o.t_lo + (uint32_t)(8 * step), b, o.b_top, ID_LO);
        else mma_ss_more(t_acc + (uint32_t)L::LO_COL0, o.r + (uint32_t)((step - lo_in_tmem) * 256), o.r_top, b, o.b_top, ID_LO);
      }
    }
  }
}

// What the parts and their three products miss of an element that is small (x: scaled), times h: hi is off by at most 2^-25, lo
// rounds that to 2^-38 or 2^-12 of itself, and lo * lo, 2^-12 of it, is left out.
__device__ __forceinline__ float part_error(float x) {
  const float m = fabsf(x);
  return fminf(m, fmaf(fminf(m, 0x1p-25f), 0x1p-11f, 0x1p-38f));
}
// That for an element of R, to be added for h = h_hi + its low part: r h - (hi h + lo h_hi).
struct Missing {
  float rest, lo;      // r - hi, lo; unscaled
};
__device__ __forceinline__ Missing missing_of(float r, float r_limit, float scale, float unscale) {
  if (!is_small(r, r_limit)) return {0.f, 0.f};
  if (!(r_limit > 0.f)) return {r, 0.f};                           // all of its row is left out
  __half hi, lo;
  split_half(r * scale, &hi, &lo);
  return {r - __half2float(hi) * unscale, __half2float(lo) * (LO_UNSCALE * unscale)};
}

// Whether what the parts miss (`error`: 2^24 times at most that) may show in a sum: above 2^-24 of it, or of 0.5 where the sum goes
// into a sigmoid.
__device__ __forceinline__ bool shows(float sum, float error) {
  return !(error <= fmaxf(fabsf(sum), (threadIdx.x & 3) != 3 ? 0.5f : 0.f));
}

// A gate row's sums for 4 NG batch rows with what the parts miss of the row's small elements, where it may show.  h of the first step
// is h0, whose own small elements are not in the parts at all.  (Rarely reached: by values, so that the step's sums stay in registers.)
template <int NG>
struct Sums {
  float v[NG][4];
};
template <int NG, typename L>
__device__ __noinline__ Sums<NG> with_missing(Sums<NG> s, const LocalArgs& a, const LocalShared* sh, const unsigned char* smem, int t) {
  const int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3, half = threadIdx.x >> 7, row = quarter * 32 + lane;
  const int b0 = (int)(blockIdx.x / (unsigned)a.cs) * a.per, nb = min(a.per, a.B - b0);
  const int unit = (int)(blockIdx.x % (unsigned)a.cs) * UNITS + row / 4, width = unit < a.H ? a.H : 0;
  const float* r_row = a.R + ((size_t)(row & 3) * a.H + (width ? unit : 0)) * a.H;
  const float m = row_magnitude(sh->row_max[row]), r_limit = limit_of(m), error = error_of(sh->row_max[row]);
  const float r_scale = pow2(scale_exponent(m)), r_unscale = pow2(-scale_exponent(m));
  const unsigned int *r_units = sh->small_r[quarter], *h0_units = sh->small_h0;
  const bool h0_small = t == 0 && nonzero_words(h0_units);
#pragma unroll
  for (int g = 0; g < NG; g++) {
    const int b = 8 * g + 4 * half;
    uint32_t want = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float e = t == 0 ? error * H_SCALE * sh->h0_unscale[b + j] : error;                      // (|h| is below 1, h0 below that)
      if (b + j < nb && (h0_small || shows(s.v[g][j], e))) want |= 1u << j;
    }
    if (!want) continue;
    if (t > 0 && !mbar_wait(smem_u32(&sh->full[t & 1]), (uint32_t)((t - 1) >> 1) & 1u, a, 96)) break;   // (this thread reads the others' words itself)
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    for (int w8 = 0; w8 < 4 * a.cs; w8++) {                        // eight units: 32 bytes of a row, together
      const uint32_t of_h0 = t == 0 ? h0_units[w8 >> 2] >> (w8 & 3) * 8 & 0xffu : 0u, units = (r_units[w8 >> 2] >> (w8 & 3) * 8 & 0xffu) | of_h0;
      if (!units) continue;
      float r[8];
#pragma unroll
      for (int i = 0; i < 8; i += 4)                               // (H is a multiple of 4, rows are 16-byte aligned)
        *reinterpret_cast<float4*>(r + i) = w8 * 8 + i < width ? *reinterpret_cast<const float4*>(r_row + w8 * 8 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      const unsigned char* p = smem + (t & 1 ? L::BUF : 0) + (L::ZERO + g) * L::GROUP + half * 64 + (w8 >> 2) * L::SRC + (w8 & 3) * 128;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (!(units >> i & 1u)) continue;
        const Missing q = missing_of(r[i], r_limit, r_scale, r_unscale);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          float unscale = H_UNSCALE;
          if (t == 0) {
            if (b + j >= nb) continue;
            unscale = sh->h0_unscale[b + j];
            if (of_h0 >> i & 1u) {
              const float h = w8 * 8 + i < width ? a.h0[(size_t)(b0 + b + j) * a.H + w8 * 8 + i] : 0.f;
              if (is_small(h, unscale > 0.f ? unscale * SMALL : __uint_as_float(0x7fffffffu))) {
                sum[j] = fmaf(r[i], h, sum[j]);
                continue;
              }
            }
          }
          const float h_hi = __half2float(*reinterpret_cast<const __half*>(p + j * 16 + i * 2)) * unscale;
          const float h_lo = __half2float(*reinterpret_cast<const __half*>(p + NG * L::GROUP + j * 16 + i * 2)) * (LO_UNSCALE * unscale);
          if (is_small(r[i], r_limit)) sum[j] = fmaf(-q.lo, h_hi, fmaf(q.rest, h_hi + h_lo, sum[j]));
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) s.v[g][j] += want >> j & 1u ? sum[j] : 0.f;
  }
  return s;
}

// The gates of GROUPS of a thread's NG cells (side by side: their chains of dependent operations overlap), h into `out`.
template <int NG, int GROUPS>
__device__ __forceinline__ void step_end(const float (&s)[NG][4], bool product, const float (&pin)[NG][4], const float (&bsum)[4],
                                         const bool (&live)[NG], float (&c)[NG], float (&h)[NG], unsigned char* out) {
  const bool up = (threadIdx.x & 2) != 0, odd = (threadIdx.x & 1) != 0;
  float w[GROUPS][4] = {};
  if (product) {
    // a unit's four lanes hold a gate each of four batch rows: turned so that each holds four gates of a row
    float x[GROUPS][2], r[GROUPS][2];
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
      r[g][0] = __shfl_xor_sync(0xffffffffu, up ? s[g][0] : s[g][2], 2);
      r[g][1] = __shfl_xor_sync(0xffffffffu, up ? s[g][1] : s[g][3], 2);
    }
#pragma unroll
    for (int g = 0; g < GROUPS; g++) {
      const float x00 = up ? r[g][0] : s[g][0], x01 = up ? r[g][1] : s[g][1], x10 = up ? s[g][2] : r[g][0], x11 = up ? s[g][3] : r[g][1];
      x[g][0] = __shfl_xor_sync(0xffffffffu, odd ? x00 : x01, 1);
      x[g][1] = __shfl_xor_sync(0xffffffffu, odd ? x10 : x11, 1);
      w[g][0] = odd ? x[g][0] : x00;
      w[g][1] = odd ? x01 : x[g][0];
      w[g][2] = odd ? x[g][1] : x10;
      w[g][3] = odd ? x11 : x[g][1];
    }
  }
#pragma unroll
  for (int g = 0; g < GROUPS; g++) {
    const float it = sigmoid_of(w[g][0] + (pin[g][0] + bsum[0])), ot = sigmoid_of(w[g][1] + (pin[g][1] + bsum[1]));
    const float ft = sigmoid_of(w[g][2] + (pin[g][2] + bsum[2])), ct = tanh_of(w[g][3] + (pin[g][3] + bsum[3]));
    c[g] = ft * c[g] + it * ct;
    h[g] = live[g] ? ot * tanh_of(c[g]) : 0.f;
  }
#pragma unroll
  for (int g = 0; g < GROUPS; g++) {
    __half hi, lo;
    split_half(h[g] * H_SCALE, &hi, &lo);
    *reinterpret_cast<__half*>(out + g * 128) = hi;
    *reinterpret_cast<__half*>(out + g * 128 + 64) = lo;
  }
}

template <int NG, int ACCS, bool TURNS>
__global__ void __launch_bounds__(THREADS, 1) lstm_local_kernel(const __grid_constant__ LocalArgs a) {
  using L = LocalLayout<NG, ACCS, TURNS>;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ LocalShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cs = a.cs, H = a.H;
  const int rank = (int)(blockIdx.x % (unsigned)cs), cluster = (int)(blockIdx.x / (unsigned)cs);
  const int b0 = cluster * a.per, nb = min(a.per, a.B - b0);
  const int u0 = rank * UNITS;
  const uint32_t buf_bytes = (uint32_t)L::BUF;
  unsigned char* stage = smem + 2 * buf_bytes;
  unsigned char* r_lo = stage + L::STAGE;                          // low parts of R past tensor memory: 4 KB a k step

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.mma_bar)));
    for (int i = 0; i < 2; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sh.full[i])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 4 * MAX_CS) sh.small_r[tid / MAX_CS][tid % MAX_CS] = 0;
  if (tid < MAX_CS) sh.small_h0[tid] = 0;
  if (tid < 8 * MAX_GROUPS) sh.h0_unscale[tid] = 1.f;
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (!a.r_early) pdl_grid_wait();

  // Gate row r of the CTA = gate r % 4 of unit r / 4.  Its largest magnitude: eight lanes take 128 consecutive bytes of a
  // row, a warp its rows 16 w .. 16 w + 15 (a thread per row, 16 bytes each, took 10 us more at 512 units).
  const int row = (warp & 3) * 32 + lane, half = warp >> 2;
  if (warp < 8) {
    for (int i = 0; i < 4; i++) {
      const int r = warp * 16 + 4 * i + lane / 8, unit = u0 + r / 4, k1 = unit < H ? H : 0;
      const float* src = a.R + ((size_t)(r & 3) * H + unit) * H;
      uint32_t m = 0;                                              // (magnitudes compare like their bits)
      for (int k = (lane & 7) * 4; k < k1; k += 256) {
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
          v[j] = k + 32 * j < k1 ? *reinterpret_cast<const uint4*>(src + k + 32 * j) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int j = 0; j < 8; j++)
          m = max(max(max(v[j].x & 0x7fffffffu, v[j].y & 0x7fffffffu), max(v[j].z & 0x7fffffffu, v[j].w & 0x7fffffffu)), m);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((lane & 7) == 0) sh.row_max[r] = __uint_as_float(m);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem_base;
  const uint32_t tmem_hi = tmem + (uint32_t)L::D_COLS, tmem_lo = tmem_hi + (uint32_t)(16 * cs);
  const int steps_lo = L::steps_lo(cs);
  float unscale = 0.f;
  if (warp < 8) {
    const float m = sh.row_max[row];
    const bool whole_row = not_finite(m);
    const int e = scale_exponent(m);
    const float r_limit = limit_of(m), scale = pow2(e);
    float row_error = 0.f;
    unscale = pow2(-e) * H_UNSCALE;                                // (e <= 100: a normal number)
    const uint32_t t_row = (uint32_t)((warp & 3) * 32) << 16;
    // 64 columns at a time through shared memory (rows 272 bytes apart: no bank conflicts either way); warps w and w + 4 take
    // 32 of them each of the rows 32 w .. 32 w + 31
    float4* chunk = reinterpret_cast<float4*>(smem + 2 * buf_bytes - 128 * 272);
    float4 next[8];
    auto fetch = [&](int k) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int r = j * 16 + tid / 16, unit = u0 + r / 4, col = k + (tid & 15) * 4;
        next[j] = unit < H && col < H ? *reinterpret_cast<const float4*>(a.R + ((size_t)(r & 3) * H + unit) * H + col)
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    fetch(0);
    for (int k = 0; k < cs * 32; k += 64) {
#pragma unroll
      for (int j = 0; j < 8; j++) chunk[(j * 16 + tid / 16) * 17 + (tid & 15)] = next[j];
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (k + 64 < cs * 32) fetch(k + 64);
      for (int i = 0; i < 2; i++) {
        const int j = k / 16 + half * 2 + i;                       // k step of 16
        if (j >= 2 * cs) break;
        uint32_t hi[8], lo[8], units = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float4 v = chunk[row * 17 + half * 8 + i * 4 + q];
          const float x[4] = {v.x, v.y, v.z, v.w};
          __half h[4], l[4];
#pragma unroll
          for (int c = 0; c < 4; c++) {
            split_half(whole_row ? 0.f : x[c] * scale, &h[c], &l[c]);
            if (is_small(x[c], r_limit)) {
              units |= 1u << (q * 4 + c);
              row_error += part_error(x[c] * scale);
            }
          }
#pragma unroll
          for (int c = 0; c < 2; c++) {
            hi[q * 2 + c] = (uint32_t)__half_as_ushort(h[2 * c]) | (uint32_t)__half_as_ushort(h[2 * c + 1]) << 16;
            lo[q * 2 + c] = (uint32_t)__half_as_ushort(l[2 * c]) | (uint32_t)__half_as_ushort(l[2 * c + 1]) << 16;
          }
        }
        if (units) atomicOr(&sh.small_r[warp & 3][j >> 1], units << (j & 1) * 16);
        tmem_st8(tmem_hi + t_row + (uint32_t)(8 * j), hi);
        if (TURNS ? (j & 1) == 0 : j < steps_lo) {
          tmem_st8(tmem_lo + t_row + (uint32_t)(8 * (TURNS ? j >> 1 : j)), lo);
        } else {
          unsigned char* dst = r_lo + (size_t)(TURNS ? j >> 1 : j - steps_lo) * 4096 + row * 16;
          *reinterpret_cast<uint4*>(dst) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(dst + 2048) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    // what the parts miss of a row's small elements, of both warps
    float* errors = reinterpret_cast<float*>(chunk);
    if (half == 1) errors[row] = row_error;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (half == 0) sh.row_max[row] = pack_row(m, (row_error + errors[row]) * pow2(-e));
  }
  __syncthreads();
  for (uint32_t i = (uint32_t)tid * 16u; i < 2u * buf_bytes; i += THREADS * 16u)   // rows past the batch stay zero
    *reinterpret_cast<uint4*>(smem + i) = make_uint4(0, 0, 0, 0);
  __syncthreads();
  if (a.r_early) pdl_grid_wait();

  // Cells of a thread: unit 8 (warp % 4) + lane / 4, batch rows 8 g + 4 (warp / 4) + lane % 4
  const int unit = u0 + 8 * (warp & 3) + lane / 4, row0 = 4 * half + (lane & 3);
  float c_reg[NG], h_reg[NG], bsum[4], pin[NG][4];
  bool live[NG];
#pragma unroll
  for (int g = 0; g < 4; g++) bsum[g] = warp < 8 && unit < H && a.bias ? a.bias[g * H + unit] + a.bias[(4 + g) * H + unit] : 0.f;
  const float* p_src = a.P + (size_t)(b0 + row0) * 4 * H + unit;
  float* y_dst = a.Y + (size_t)(b0 + row0) * H + unit;
#pragma unroll
  for (int g = 0; g < NG; g++) {
    live[g] = warp < 8 && unit < H && 8 * g + row0 < nb;
    c_reg[g] = live[g] && a.c0 ? a.c0[(size_t)(b0 + 8 * g + row0) * H + unit] : 0.f;
    h_reg[g] = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) pin[g][q] = live[g] ? p_src[(size_t)8 * g * 4 * H + q * H] : 0.f;
  }
  constexpr int HI_OFF = L::ZERO * L::GROUP, LO_OFF = HI_OFF + NG * L::GROUP;
  if (a.h0) {   // into buffer 0, each batch row with a scale of its own
    for (int b = warp; b < nb; b += THREADS / 32) {
      const float* src = a.h0 + (size_t)(b0 + b) * H;
      uint32_t m = 0;
      for (int k = lane; k < H; k += 32) m = max(m, __float_as_uint(src[k]) & 0x7fffffffu);
      m = __reduce_max_sync(0xffffffffu, m);
      const int e = scale_exponent(__uint_as_float(m));
      const float scale = pow2(e), limit = limit_of(__uint_as_float(m));
      if (lane == 0) sh.h0_unscale[b] = limit > 0.f ? pow2(-e) : -1.f;
      for (int k = lane; k < H; k += 32) {
        __half hi, lo;
        const bool small = is_small(src[k], limit);
        split_half(small ? 0.f : src[k] * scale, &hi, &lo);
        if (small) atomicOr(&sh.small_h0[k >> 5], 1u << (k & 31));
        unsigned char* p = smem + (k >> 5) * L::SRC + (b >> 3) * 512 + ((k >> 3) & 3) * 128 + (b & 7) * 16 + (k & 7) * 2;
        *reinterpret_cast<__half*>(p + HI_OFF) = hi;
        *reinterpret_cast<__half*>(p + LO_OFF) = lo;
      }
    }
  }
  const uint32_t full0 = smem_u32(&sh.full[0]);
  const int quarters = (cs + 3) / 4;
  const uint32_t step_bytes = (uint32_t)cs * (uint32_t)nb * 128u + a.beyond;  // a source sends 128 for each batch row
  if (tid == 0) {
    expect_bytes(full0, step_bytes);
    expect_bytes(full0 + 8u, step_bytes);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // (zeros, h0 and low parts of R are read by the MMAs)
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();                                               // every CTA is ready for the others' words
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t small_r = nonzero_words(sh.small_r[warp & 3]), small_h0 = nonzero_words(sh.small_h0);
  const uint32_t mma_bar = smem_u32(&sh.mma_bar);

  if (warp == 8) {
    const uint64_t b_desc = make_desc(smem_u32(smem), 128, L::GROUP), r_desc = make_desc(smem_u32(r_lo), 2048, 128);
    if (elect_one()) {
      for (int t = a.h0 ? 0 : 1; t < a.T; t++) {
        const uint32_t bar = full0 + (t & 1 ? 8u : 0u);
        if (t > 0) {
          if (!mbar_wait(bar, (uint32_t)((t - 1) >> 1) & 1u, a, 94)) break;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int q = 0; q < quarters; q++) {
          const int n = cs - 4 * q, lo_in_tmem = steps_lo - 8 * q;
          const Issue o = {tmem, tmem_hi + (uint32_t)(64 * q), tmem_lo + (uint32_t)((TURNS ? 32 : 64) * q),
                           (uint32_t)b_desc + (uint32_t)(((t & 1) * L::BUF + 4 * q * L::SRC) >> 4), (uint32_t)(b_desc >> 32),
                           (uint32_t)r_desc + (TURNS ? (uint32_t)(1024 * q) : 0u), (uint32_t)(r_desc >> 32)};
          if (n >= 4 && (TURNS || lo_in_tmem >= 8)) issue_sources<NG, ACCS, TURNS, true>(o, q, n, lo_in_tmem);
          else issue_sources<NG, ACCS, TURNS, false>(o, q, n, lo_in_tmem);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mma_bar) : "memory");
        if (t > 0) expect_bytes(bar, step_bytes);                  // the words of step t + 2
      }
    }
    __syncwarp();
  } else {
    const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(4 * half);
    // words on their way out: [group][hi, lo][4 batch rows][8 units] of this warp
    unsigned char* out = stage + warp * (128 * NG);
    unsigned char* my_out = out + (lane & 3) * 16 + (lane >> 2) * 2;
    const int w_part = (lane >> 2) & 1, w_row = lane & 3, dist = lane >> 3;
    uint32_t dst[QUARTERS];
    uint32_t reach = 0;                                            // which of its up to four receivers there are
    const uint32_t my_slot = smem_u32(smem) + (uint32_t)(rank * L::SRC + (w_part ? LO_OFF : HI_OFF) + (warp & 3) * 128 + (4 * half + w_row) * 16);
    const uint32_t to_bar = full0 - my_slot;                       // from where the word goes to its barrier
#pragma unroll
    for (int i = 0; i < QUARTERS; i++) {
      int peer = rank + dist + 4 * i;                              // (not all CTAs start with the same receiver)
      if (dist + 4 * i < cs) reach |= 1u << i;
      if (peer >= cs) peer -= cs;
      dst[i] = map_to(my_slot, (uint32_t)(dist + 4 * i < cs ? peer : rank));
    }
    const bool some = 4 * half < nb;                               // (the last rows' warps may have nothing to do)
    const bool last_empty = 8 * (NG - 1) + 4 * half >= nb;
    uint32_t phase = 0;
    for (int t = 0; t < a.T && some; t++) {
      float s[NG][4];
      const bool product = t > 0 || a.h0;
      if (product) {
        if (!__all_sync(0xffffffffu, mbar_wait(mma_bar, phase, a, 95))) break;
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float x[NG][4];
        constexpr int PART = NG == 1 ? ACCS : NG == 2 && ACCS % 2 == 0 ? 2 : 1;   // accumulators read at once
#pragma unroll
        for (int i = 0; i < ACCS; i += PART) {
          float hh[PART][NG][4], cross[PART][NG][4];
#pragma unroll
          for (int p = 0; p < PART; p++)
#pragma unroll
            for (int g = 0; g < NG; g++) {
              tmem_ld4(t_row + (uint32_t)((i + p) * L::ACC + 8 * g), hh[p][g]);
              tmem_ld4(t_row + (uint32_t)((i + p) * L::ACC + 8 * NG + 8 * g), cross[p][g]);
            }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int p = 0; p < PART; p++)
#pragma unroll
            for (int g = 0; g < NG; g++)
#pragma unroll
              for (int j = 0; j < 4; j++) {
                s[g][j] = i + p ? s[g][j] + hh[p][g][j] : hh[p][g][j];
                x[g][j] = i + p ? x[g][j] + cross[p][g][j] : cross[p][g][j];
              }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
#pragma unroll
        for (int g = 0; g < NG; g++)
#pragma unroll
          for (int j = 0; j < 4; j++) s[g][j] = fmaf(x[g][j], LO_UNSCALE, s[g][j]) * unscale;
        if (t == 0) {                                              // h0 has scales of its own
#pragma unroll
          for (int g = 0; g < NG; g++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[g][j] = s[g][j] * H_SCALE * sh.h0_unscale[8 * g + 4 * half + j];
        }
        if (t == 0 ? small_r | small_h0 : small_r) {
          const float error = error_of(sh.row_max[row]);
          bool some_show = t == 0;                                 // (asked there)
#pragma unroll
          for (int i = 0; i < 4 * NG; i++) some_show |= i / 4 * 8 + 4 * half + i % 4 < nb && shows(s[i / 4][i % 4], error);
          if (some_show) {
            Sums<NG> all;
#pragma unroll
            for (int i = 0; i < 4 * NG; i++) all.v[i / 4][i % 4] = s[i / 4][i % 4];
            all = with_missing<NG, L>(all, a, &sh, smem, t);
#pragma unroll
            for (int i = 0; i < 4 * NG; i++) s[i / 4][i % 4] = all.v[i / 4][i % 4];
          }
          __syncwarp();
        }
      }
      // (the last group of a warp's rows may be empty: a branch for all of its threads)
      if (NG > 1 && last_empty) step_end<NG, (NG > 1 ? NG - 1 : 1)>(s, product, pin, bsum, live, c_reg, h_reg, my_out);
      else step_end<NG, NG>(s, product, pin, bsum, live, c_reg, h_reg, my_out);
      __syncwarp();
      if (t + 1 < a.T) {
        const uint32_t to = t & 1 ? 0u : buf_bytes, bar = to_bar + (t & 1 ? 0u : 8u);   // buffer and barrier of step t + 1
#pragma unroll
        for (int g = 0; g < NG; g++) {
          if (8 * g + 4 * half + w_row < nb) {
            const uint4 v = *reinterpret_cast<const uint4*>(out + g * 128 + (lane & 7) * 16);
#pragma unroll
            for (int i = 0; i < QUARTERS; i++)
              if (reach >> i & 1u) send16(dst[i] + to + (uint32_t)(g * L::GROUP), dst[i] + bar, v);
          }
        }
        __syncwarp();
      }
      p_src += (size_t)a.B * 4 * H;
#pragma unroll
      for (int g = 0; g < NG; g++) {
        if (!live[g]) continue;
        y_dst[(size_t)8 * g * H] = h_reg[g];
        if (t + 1 < a.T) {
#pragma unroll
          for (int q = 0; q < 4; q++) pin[g][q] = p_src[(size_t)8 * g * 4 * H + q * H];
        }
      }
      y_dst += (size_t)a.B * H;
    }
#pragma unroll
    for (int g = 0; g < NG; g++) {
      if (!live[g]) continue;
      a.Yh[(size_t)(b0 + 8 * g + row0) * H + unit] = h_reg[g];
      a.Yc[(size_t)(b0 + 8 * g + row0) * H + unit] = c_reg[g];
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();
  if (warp == 8) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

typedef void (*Kernel)(const LocalArgs);

struct Variant {
  Kernel kernel;
  int d_cols, buf, stage;
  bool turns;
};
template <int NG, int ACCS, bool TURNS>
constexpr Variant variant() {
  using L = LocalLayout<NG, ACCS, TURNS>;
  return {lstm_local_kernel<NG, ACCS, TURNS>, L::D_COLS, L::BUF, L::STAGE, TURNS};
}
const Variant variants[MAX_GROUPS][2] = {   // [8-row groups - 1][more than one CTA a cluster]
    {variant<1, 2, false>(), variant<1, 4, false>()}, {variant<2, 2, false>(), variant<2, 4, false>()},
    {variant<3, 2, false>(), variant<3, 4, false>()}, {variant<4, 2, false>(), variant<4, 4, false>()}};
const Variant two_groups_in_turns = variant<2, 4, true>();

// k steps whose low parts of R are in shared memory
int steps_in_smem(const Variant& v, int cs) {
  const int steps = 4 * cs - (512 - v.d_cols) / 8;
  return v.turns ? cs : steps < 0 ? 0 : steps;
}
size_t smem_of(const Variant& v, int cs) {
  const size_t bytes = 2 * (size_t)v.buf + v.stage + (size_t)steps_in_smem(v, cs) * 4096;
  return bytes < MIN_SMEM ? MIN_SMEM : bytes;
}

// Four accumulators, or one for each k step where there are two.  Two groups of rows on 15 and 16 CTAs have 12 and 16 k steps in
// shared memory, and take every other one there: a step of [64, 480] 2.32 -> 2.28 us, of [64, 512] 2.47 -> 2.38 (with 8 of them, one
// group on 16 CTAs, it is the other way round, 1.33 and 1.38, as there would be 16).
const Variant& variant_of(int groups, int cs) {
  const Variant& v = variants[groups - 1][cs > 1];
  return groups == 2 && steps_in_smem(v, cs) > 8 ? two_groups_in_turns : v;
}
// 8-row groups of a cluster, at most: with four, 14 CTAs and more have no room for the low parts of R.
int max_groups(int cs) { return cs <= 13 ? MAX_GROUPS : MAX_GROUPS - 1; }

void fill_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int grid, int cs, size_t smem, cudaStream_t stream) {
  *cfg = {};
  cfg->gridDim = dim3((unsigned)grid);
  cfg->blockDim = dim3(THREADS);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}

// Clusters that can be resident at once (asked once per device and shape).
int max_clusters(wdc_context* ctx, int cs, const Variant& v) {
  static std::mutex mu;
  static std::map<std::pair<std::pair<int, int>, Kernel>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(std::make_pair(ctx->device, cs), v.kernel);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(v.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  fill_config(&cfg, attr, cs, cs, smem_of(v, cs), nullptr);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, v.kernel, &cfg);
  if (e != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known[key] = n;
  return n;
}

}  // namespace

// Runs the recurrence on the projected input P.  WDC_ERR_UNSUPPORTED: shape outside the kernel's range (nothing has been
// written); any other non-zero status is an error.
int wdc_lstm_local(wdc_context* ctx, const float* P, const float* R, const float* bias, const float* h0, const float* c0,
                   float* Y, float* Yh, float* Yc, int64_t T, int64_t Bt, int64_t H, int64_t selftest_wait_ns) {
  if (T < 4 || H < UNITS || H > MAX_CS * UNITS || H % 4 != 0) return WDC_ERR_UNSUPPORTED;
  if (T > (1 << 24) || Bt > (1 << 20)) return WDC_ERR_UNSUPPORTED;
  if (((uintptr_t)R & 15) != 0) return WDC_ERR_UNSUPPORTED;
  LocalArgs a = {P, R, bias, h0, c0, Y, Yh, Yc, ctx->status_word, (int)T, (int)Bt, (int)H};
  a.cs = (int)((H + UNITS - 1) / UNITS);
  const int fit = max_clusters(ctx, a.cs, variant_of(max_groups(a.cs), a.cs));
  if (!fit) return WDC_ERR_UNSUPPORTED;
  const int64_t rounds = ceil_div64(Bt, (int64_t)fit * 8 * max_groups(a.cs));
  a.per = (int)ceil_div64(Bt, rounds * fit);
  const int groups = (a.per + 7) / 8, clusters = (int)ceil_div64(Bt, a.per);
  const Variant& v = variant_of(groups, a.cs);
  if (!max_clusters(ctx, a.cs, v)) return WDC_ERR_UNSUPPORTED;
  a.beyond = selftest_wait_ns > 0 ? 16u : 0u;
  a.wait_ns = selftest_wait_ns > 0 ? (unsigned long long)selftest_wait_ns : WAIT_NS;
  // A declared constant may have been written by the grid in front of the projection's: every kernel of the projection waits
  // for the grids in front of it before it lets the next one start, so that one has finished by now.  (Only the projection,
  // which is always launched in between, may still be running.)
  a.r_early = ctx->opt_pdl && wdc_is_constant(ctx, R);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  fill_config(&cfg, attr, clusters * a.cs, a.cs, smem_of(v, a.cs), ctx->stream);
  cfg.numAttrs = ctx->opt_pdl ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, v.kernel, (const LocalArgs)a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return WDC_ERR_UNSUPPORTED;
  }
  ctx->n_tc_launch++;
  return wdc_check_launch(ctx, "lstm_local_kernel");
}
