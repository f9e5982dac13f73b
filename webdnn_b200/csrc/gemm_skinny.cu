// Gemm with few rows of A (a single request, a handful of them): Y[m, n] = alpha * A[m, :] . B[:, n] + beta * C[m, n].
//
// Bound by reading B once (4 bytes for 2 * m FLOP) and, at the sizes such layers have, by latency: a 128-row
// tensor-core tile would be nearly empty, and the 64x64 CUDA-core tiles of gemm_simt.cu put 2048x1000 on 16 CTAs
// with 128 dependent K steps (334 us for [1, 2048] x [2048, 1000]; a ResNet-50 run of one image, whose last layer this
// is, went from 958 to 633 us, the 784-512-512-10 MLP on one row from 206 to 41 us).  Here the whole chip reads B at once and every
// thread has its loads in flight together:
//   * B stored [n][k] (Gemm transB = 1): a warp takes NC columns and one slice of K, 16 bytes per lane and column;
//     `wk` warps of the CTA share a column group and split K, so that most layers are one round trip of loads;
//   * B stored [k][n] (MatMul, transB = 0): a lane owns one column (coalesced rows of B), the CTA's 16 warps split K.
// MT rows of A are kept per CTA (grid.y walks the rest; B then comes from L2).  fp32 FMAs; the partial sums of lanes
// and warps are added in a fixed order.
#include "common.cuh"

namespace {

constexpr int NC = 4;            // columns per warp
constexpr int ROW_WARPS = 8;     // warps per CTA, B stored [n][k]
constexpr int COL_WARPS = 16;    // warps per CTA, B stored [k][n]
constexpr int COL_UNROLL = 8;    // rows of B a lane has in flight

struct SkinnyArgs {
  const float* A;
  const float* B;
  const float* C;                // null: no addend
  float* Y;
  int64_t sab, sa0, sa1, sbb, sb, sc0, sc1;   // sb: pitch of the stored rows of B
  int64_t m, n, k;
  float alpha, beta;
  int relu;
};

__device__ __forceinline__ void store_out(const SkinnyArgs& a, int64_t bz, int64_t m, int64_t n, float v) {
  v *= a.alpha;
  if (a.C) v += pdl_ld(pdl_after(a.C) + m * a.sc0 + n * a.sc1) * a.beta;
  if (a.relu) v = v > 0.f ? v : (v == v ? 0.f : v);
  a.Y[(bz * a.m + m) * a.n + n] = v;
}

// Sum of v[0..COUNT) over the warp, spread so that lane l ends up with the total of v[l % COUNT]: COUNT - 1 shuffles
// while the values halve, then plain butterfly steps, instead of 5 * COUNT.
template <int COUNT>
__device__ __forceinline__ float spread_sum(float* v, int lane) {
#pragma unroll
  for (int half = COUNT / 2, off = 16; half >= 1; half >>= 1, off >>= 1) {
    // lanes with bit `off` set keep the upper half of the values
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const float send = up ? v[i] : v[i + half];
      const float keep = up ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  float s = v[0];
#pragma unroll
  for (int off = 16 / COUNT; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}
// Which value of spread_sum a lane holds: bit 4 of the lane chose the top half first, and so on downwards.
template <int COUNT>
__device__ __forceinline__ int spread_index(int lane) { return lane / (32 / COUNT); }

// B stored [n][k].  grid: (ceil(n / (NC * ROW_WARPS / wk)), ceil(m / MT), batch); wk warps split K.
template <int MT, int VEC>
__global__ void __launch_bounds__(ROW_WARPS * 32) skinny_rows_kernel(const SkinnyArgs a, int wk) {
  pdl_wait();
  __shared__ float red[ROW_WARPS][MT * NC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kw = warp % wk, group = warp / wk, groups = ROW_WARPS / wk;
  const int64_t n0 = ((int64_t)blockIdx.x * groups + group) * NC;
  const int64_t m0 = (int64_t)blockIdx.y * MT, bz = blockIdx.z;
  const float* A = pdl_after(a.A) + bz * a.sab + m0 * a.sa0;
  const float* B = pdl_after(a.B) + bz * a.sbb;
  // columns and rows past the edge repeat the last valid one and are not stored
  const float* bp[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) bp[c] = B + (n0 + c < a.n ? n0 + c : a.n - 1) * a.sb;
  const float* ap[MT];
#pragma unroll
  for (int r = 0; r < MT; r++) ap[r] = A + (m0 + r < a.m ? r : a.m - 1 - m0) * a.sa0;
  float acc[MT * NC];
#pragma unroll
  for (int i = 0; i < MT * NC; i++) acc[i] = 0.f;
#pragma unroll 2
  for (int64_t k = (int64_t)(kw * 32 + lane) * VEC; k < a.k; k += (int64_t)wk * 32 * VEC) {
    if (VEC == 4) {
      float4 w[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) w[c] = pdl_ld(reinterpret_cast<const float4*>(bp[c] + k));
#pragma unroll
      for (int r = 0; r < MT; r++) {
        const float4 x = pdl_ld(reinterpret_cast<const float4*>(ap[r] + k));
#pragma unroll
        for (int c = 0; c < NC; c++) {
          float& s = acc[r * NC + c];
          s = fmaf(x.x, w[c].x, s);
          s = fmaf(x.y, w[c].y, s);
          s = fmaf(x.z, w[c].z, s);
          s = fmaf(x.w, w[c].w, s);
        }
      }
    } else {
      float w[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) w[c] = pdl_ld(bp[c] + k);
#pragma unroll
      for (int r = 0; r < MT; r++) {
        const float x = pdl_ld(ap[r] + k * a.sa1);
#pragma unroll
        for (int c = 0; c < NC; c++) acc[r * NC + c] = fmaf(x, w[c], acc[r * NC + c]);
      }
    }
  }
  const float s = spread_sum<MT * NC>(acc, lane);
  if (lane % (32 / (MT * NC)) == 0) red[warp][spread_index<MT * NC>(lane)] = s;
  __syncthreads();
  for (int i = threadIdx.x; i < groups * MT * NC; i += ROW_WARPS * 32) {
    const int g = i / (MT * NC), e = i - g * (MT * NC), r = e / NC, c = e % NC;
    const int64_t n = ((int64_t)blockIdx.x * groups + g) * NC + c;
    float v = 0.f;
    for (int w = 0; w < wk; w++) v += red[g * wk + w][e];
    if (m0 + r < a.m && n < a.n) store_out(a, bz, m0 + r, n, v);
  }
}

// B stored [k][n].  grid: (ceil(n / 32), ceil(m / MT), batch); the warps take rows w, w + 16, ... of B.
template <int MT>
__global__ void __launch_bounds__(COL_WARPS * 32) skinny_cols_kernel(const SkinnyArgs a) {
  pdl_wait();
  __shared__ float red[COL_WARPS][MT][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t n = (int64_t)blockIdx.x * 32 + lane;
  const int64_t m0 = (int64_t)blockIdx.y * MT, bz = blockIdx.z;
  const float* A = pdl_after(a.A) + bz * a.sab + m0 * a.sa0;
  const float* bp = pdl_after(a.B) + bz * a.sbb + (n < a.n ? n : a.n - 1);
  const int rows = a.m - m0 < MT ? (int)(a.m - m0) : MT;
  float acc[MT];
#pragma unroll
  for (int r = 0; r < MT; r++) acc[r] = 0.f;
  for (int64_t k0 = warp; k0 < a.k; k0 += COL_WARPS * COL_UNROLL) {
    float w[COL_UNROLL];
#pragma unroll
    for (int j = 0; j < COL_UNROLL; j++) {
      const int64_t k = k0 + j * COL_WARPS;
      w[j] = k < a.k ? pdl_ld(bp + k * a.sb) : 0.f;
    }
    // lane j of the warp fetches A[r][k0 + 16 j]: one load per row, handed round by shuffles
#pragma unroll
    for (int r = 0; r < MT; r++) {
      const int64_t k = k0 + (lane % COL_UNROLL) * COL_WARPS;
      const float x = (r < rows && k < a.k) ? pdl_ld(A + r * a.sa0 + k * a.sa1) : 0.f;
#pragma unroll
      for (int j = 0; j < COL_UNROLL; j++)
        if (k0 + j * COL_WARPS < a.k) acc[r] = fmaf(__shfl_sync(0xffffffffu, x, j), w[j], acc[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < MT; r++) red[warp][r][lane] = acc[r];
  __syncthreads();
  for (int i = threadIdx.x; i < rows * 32; i += COL_WARPS * 32) {
    const int r = i >> 5, c = i & 31;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < COL_WARPS; w++) v += red[w][r][c];
    const int64_t nn = (int64_t)blockIdx.x * 32 + c;
    if (nn < a.n) store_out(a, bz, m0 + r, nn, v);
  }
}

template <int MT>
void launch_rows(wdc_context* ctx, const SkinnyArgs& a, dim3 grid, int wk, bool vec) {
  if (vec) wdc_launch_pdl(ctx, skinny_rows_kernel<MT, 4>, grid, dim3(ROW_WARPS * 32), 0, a, wk);
  else wdc_launch_pdl(ctx, skinny_rows_kernel<MT, 1>, grid, dim3(ROW_WARPS * 32), 0, a, wk);
}

}  // namespace

// Few-row Gemm.  WDC_ERR_UNSUPPORTED (nothing written): the strides of B fit neither kernel, or the grid would not.
int wdc_skinny_gemm(wdc_context* ctx, const wdc_gemm_desc* d, const float* A, const float* B, const float* C, float* Y) {
  const bool k_major = d->sb0 == 1, n_major = d->sb1 == 1;
  if (!k_major && !n_major) return WDC_ERR_UNSUPPORTED;
  if (d->batch > 65535 || d->n > (1ll << 30)) return WDC_ERR_UNSUPPORTED;
  SkinnyArgs a = {A, B, C, Y, d->sab, d->sa0, d->sa1, d->sbb, k_major ? d->sb1 : d->sb0, d->sc0, d->sc1,
                  d->m, d->n, d->k, d->alpha, d->beta, d->relu};
  // 8 rows per CTA keep the accumulators (8 x 4) in registers; fewer where there are fewer
  const int mt = d->m > 4 ? 8 : d->m > 2 ? 4 : (int)d->m;
  const unsigned gy = (unsigned)ceil_div64(d->m, mt), gz = (unsigned)d->batch;
  if (k_major) {
    const bool vec = d->sa1 == 1 && d->k % 4 == 0 && d->sa0 % 4 == 0 && d->sab % 4 == 0 && d->sb1 % 4 == 0 &&
                     d->sbb % 4 == 0 && (((uintptr_t)A | (uintptr_t)B) & 15) == 0;
    // warps that share a column group: as many as have a first load of K to do
    int wk = 1;
    while (wk < ROW_WARPS && (int64_t)wk * 32 * (vec ? 4 : 1) < d->k) wk *= 2;
    const dim3 grid((unsigned)ceil_div64(d->n, NC * (ROW_WARPS / wk)), gy, gz);
    if (mt == 8) launch_rows<8>(ctx, a, grid, wk, vec);
    else if (mt == 4) launch_rows<4>(ctx, a, grid, wk, vec);
    else if (mt == 2) launch_rows<2>(ctx, a, grid, wk, vec);
    else launch_rows<1>(ctx, a, grid, wk, vec);
    return wdc_check_launch(ctx, "skinny_rows_kernel");
  }
  const dim3 grid((unsigned)ceil_div64(d->n, 32), gy, gz);
  if (mt == 8) wdc_launch_pdl(ctx, skinny_cols_kernel<8>, grid, dim3(COL_WARPS * 32), 0, a);
  else if (mt == 4) wdc_launch_pdl(ctx, skinny_cols_kernel<4>, grid, dim3(COL_WARPS * 32), 0, a);
  else if (mt == 2) wdc_launch_pdl(ctx, skinny_cols_kernel<2>, grid, dim3(COL_WARPS * 32), 0, a);
  else wdc_launch_pdl(ctx, skinny_cols_kernel<1>, grid, dim3(COL_WARPS * 32), 0, a);
  return wdc_check_launch(ctx, "skinny_cols_kernel");
}
