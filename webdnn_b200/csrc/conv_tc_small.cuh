// The contraction of conv_tc.cu for outputs of at most a wave or two of tiles: one image through a network, the
// layers of a transformer over a few hundred tokens.  Included by conv_tc.cu inside its namespace.
//
// Such a launch is bound by latency.  The persistent kernel takes the whole SM (512 threads x 128 registers, 218 KB,
// all of tensor memory), so a launch cannot begin its set-up while the one before it drains; its tiles walk the whole
// reduction; and a reduction cut into ranges needs a second launch.  Here
//   * a CTA computes one 128 x TN tile over one part of K and takes less than half an SM (352 threads x <= 88
//     registers, 256 TMEM columns, 96 KB of stages and, with 32 columns, up to 18 KB for the exchange): under
//     programmatic dependent launch the next launch's CTAs sit beside this one's, with barriers, tensor memory and the
//     first weight tiles ready when the wait for this one ends;
//   * the parts of a tile are the CTAs of a thread-block cluster: each sends its partial sums to the CTA that
//     finishes the row (st.async into distributed shared memory), which adds them in rank order and runs the epilogue;
//   * a barrier operation answers after 150-250 cycles whatever it finds, and one warp's operations on the way of a
//     K block add up: with separate rings for A, W and tensor memory the issuing lane's three waits and two commits
//     made a K block 1000 cycles long, of which its 12 MMAs are 200-400.  So A and W of a K block share a stage, one
//     commit frees it (for both loaders, and tensor memory for the splitters), and the issuing lane waits for one
//     barrier only.  A and W are loaded by warps of their own;
//   * warps 0-7 split A into tensor memory in two groups that take alternate K blocks, and become the epilogue.
// (The high part of A straight from its shared-memory tile would save the splitters half their work, but an MMA with
// A in shared memory took about 64 cycles whatever its width: 730-880 cycles per K block.)
// The products are those of tc_igemm_kernel, and so is the order of every addition, whatever the tile and the cluster: a
// result does not depend on which of the two kernels a launch takes.  That matters where a network carries the last bits
// on: a softmax over large scores is an argmax, and close rivals exchange places.  The parts are therefore the terms that
// kernel adds up in fp32: where it takes a tile whole, its segments of SEG_KBLOCKS K blocks, walked from the same rotated
// start and added behind the addend (rows of any length, which leave through that kernel's plain epilogue: in front of
// it); where it cuts a tile, its ranges.

constexpr int SM_SPLIT_WARPS = 8;
constexpr int SM_A_WARP = 8, SM_W_WARP = 9, SM_MMA_WARP = 10;
constexpr int SM_THREADS = 352;
constexpr int SM_EPI_THREADS = SM_SPLIT_WARPS * 32;
constexpr int SM_TMEM_COLS = 256;

// ROWS: rows of a tile that a CTA finishes, at most.
template <int TN, int CS>
struct SmallLayout {
  static constexpr int ROWS = (TILE_M + CS - 1) / CS;
  static constexpr int W_BYTES = TN * 128;                 // one of the two parts of a weight tile
  static constexpr int STAGES = TN == 64 ? 3 : 4;
  static constexpr int STAGE = A_TILE_BYTES + 2 * W_BYTES;
  static constexpr int BYTES = STAGES * STAGE;             // 96 KB
  static constexpr int BUFS = TN == 64 ? 1 : 2;            // segment accumulators
  static constexpr int T_ST = 3;                           // stages of A in tensor memory, 64 columns each
  static constexpr int A_COL0 = BUFS * TN;
  static_assert(A_COL0 + T_ST * 64 <= SM_TMEM_COLS, "tensor memory");
  static_assert(STAGES >= T_ST, "a stage's commit also frees its A in tensor memory");
  // Exchanged sums: a buffer of their own for the narrow tile; the wide tile's would not leave room for two CTAs on an
  // SM and reuses the stages, for which the cluster has to meet after its last MMA.
  static constexpr bool OWN_EXCHANGE = TN == 32;
  static constexpr int EXCHANGE_OFF = OWN_EXCHANGE ? BYTES : 0;
  static constexpr int EXCHANGE = CS * ROWS * TN * 4;
  static constexpr int SHARED_OFF = BYTES + (OWN_EXCHANGE ? EXCHANGE : 0);
  static constexpr int SMEM = SHARED_OFF + 256;            // no slack: the buffer itself is aligned (checked below)
  static_assert(EXCHANGE <= BYTES, "the exchanged sums fit the stages");
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs on an SM");
};

struct SmallShared {
  unsigned long long full[4], t_full[4], empty[4], seg_full[2], seg_empty[2];
  unsigned long long recv;
  unsigned int tmem_base;
  volatile int abort_flag;
};
static_assert(sizeof(SmallShared) <= 256, "SmallLayout::SMEM");

__device__ __noinline__ bool small_wait_slow(uint32_t bar, uint32_t parity, SmallShared* ss, int* status, int code) {
  const unsigned long long t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 1024; i++)
      if (try_wait_at(bar, parity)) return true;
    if (ss->abort_flag) return false;
    if (global_ns() - t0 > WAIT_LIMIT_NS) {
      ss->abort_flag = 1;
      atomicCAS(status, 0, code);
      return false;
    }
  }
}
__device__ __forceinline__ bool small_wait(uint32_t bar, uint32_t parity, SmallShared* ss, int* status, int code) {
  for (int i = 0; i < 4096; i++)
    if (try_wait_at(bar, parity)) return true;
  return small_wait_slow(bar, parity, ss, status, code);
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

__device__ __forceinline__ void tma_load_2d_at(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"((unsigned long long)map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_im2col_at(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c, int w, int h,
                                                   int n, int off_w, int off_h) {
  const unsigned short ow = (unsigned short)off_w, oh = (unsigned short)off_h;
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(dst),
      "l"((unsigned long long)map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n), "h"(ow), "h"(oh)
      : "memory");
}

// Where the 16-byte cell (row, cell) of one source's sums lies in the exchange buffer of a CTA that finishes ROWS rows:
// consecutive rows of a cell are consecutive words (one block per store of a warp), turned by the cell where ROWS is a
// power of two, so that a row's cells lie in different banks.
template <int ROWS>
__device__ __forceinline__ uint32_t exchange_slot(uint32_t row, uint32_t cell) {
  return cell * ROWS + (ROWS % 8 == 0 ? row ^ (cell & 7u) : row);
}

// Four columns from `n` on of a row of N; RAGGED: N is no multiple of 4, rows start anywhere, the last cell is short.
template <bool RAGGED>
__device__ __forceinline__ float4 small_cell(const float* p, int n, int N) {
  if (!RAGGED) return pdl_ld(reinterpret_cast<const float4*>(p));
  float4 v = make_float4(pdl_ld(p), 0.f, 0.f, 0.f);
  if (n + 1 < N) v.y = pdl_ld(p + 1);
  if (n + 2 < N) v.z = pdl_ld(p + 2);
  if (n + 3 < N) v.w = pdl_ld(p + 3);
  return v;
}

// CS: CTAs of a cluster = parts of K (1: the tile as a whole).  grid: tiles_m * tiles_n * CS.
// RAGGED: N is no multiple of 4.  Variants of their own: asked at run time, every launch of a network paid for the question
// (ResNet-50, one image: 428 us a run as here, 434 with it).
template <int TN, int CS, bool RAGGED>
__global__ void __launch_bounds__(SM_THREADS, 2)
tc_small_kernel(const __grid_constant__ TcProblem p, const __grid_constant__ CUtensorMap map_w_hi,
                const __grid_constant__ CUtensorMap map_w_lo, const __grid_constant__ CUtensorMap map_a,
                float* __restrict__ y, int w_early) {
  using L = SmallLayout<TN, CS>;
  constexpr int ROWS = L::ROWS;
  constexpr int CELLS = TN / 4;
  constexpr int ITEMS = (ROWS * CELLS + SM_EPI_THREADS - 1) / SM_EPI_THREADS;
  constexpr int COLS = TN / 2;                             // accumulator columns of a warp
  extern __shared__ __align__(1024) unsigned char smem_small[];
  unsigned char* smem = smem_small;
  SmallShared* ss = reinterpret_cast<SmallShared*>(smem + L::SHARED_OFF);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)(blockIdx.x % CS), tile = (int)(blockIdx.x / CS);
  const int n0 = (tile % p.tiles_n) * TN;
  const int64_t m0 = (int64_t)(tile / p.tiles_n) * TILE_M;
  // this CTA's part of the reduction (never empty): nkb K blocks from kb0 on, around the end where the tile is rotated
  const int first_kb = CS == 1 ? 0 : rank * p.part;
  const int nkb = rank == CS - 1 ? p.kblocks - first_kb : p.part;
  const int nseg = segments_of(nkb);
  int kb0 = first_kb;
  if (p.rot_grid) {
    const uint32_t whole = (uint32_t)(tile / p.tiles_n) * (uint32_t)p.rot_tiles_n + (uint32_t)(n0 % p.rot_n / p.rot_tile_n);
    kb0 += (int)(whole % (uint32_t)p.rot_grid * (uint32_t)p.kblocks / (uint32_t)p.rot_grid);
    if (kb0 >= p.kblocks) kb0 -= p.kblocks;
  }
  // the tile's rows that exist are finished in equal shares: the exchange is 16 bytes a clock, so rows past M stay out
  const int rows = p.M - m0 < TILE_M ? (int)(p.M - m0) : TILE_M;
  const int share = (rows + CS - 1) / CS;
  const int mine = rows - rank * share < 0 ? 0 : rows - rank * share < share ? rows - rank * share : share;

  {
    const int t = threadIdx.x;
    unsigned long long* bar = nullptr;
    int count = 1;
    if (t < 4) { bar = &ss->full[t]; count = 2; }
    else if (t < 8) { bar = &ss->t_full[t - 4]; count = 4; }
    else if (t < 12) bar = &ss->empty[t - 8];
    else if (t < 14) bar = &ss->seg_full[t - 12];
    else if (t < 16) { bar = &ss->seg_empty[t - 14]; count = SM_SPLIT_WARPS; }
    else if (t == 16) bar = &ss->recv;
    if (bar) {
      mbar_init(bar, count);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (t == 32) ss->abort_flag = (smem_u32(smem) & 1023u) != 0 ? 1 : 0;   // (operands are swizzled by address)
    if (t == 32 && ss->abort_flag) atomicCAS(p.status, 0, 50);
  }
  if (warp == SM_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ss->tmem_base)),
                 "r"(SM_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (warp == SM_W_WARP && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w_hi) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_w_lo) : "memory");
  }
  if (warp == SM_A_WARP && lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"((unsigned long long)&map_a) : "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (CS > 1 && L::OWN_EXCHANGE)   // this CTA's barriers are ready for the others' sums
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const uint32_t tmem_base = ss->tmem_base;
  const int q4 = warp & 3, half = warp >> 2;
  float acc[COLS];
  bool ok = true;

  if (warp < SM_SPLIT_WARPS) {
    // ============================================================================ splitters
    const uint32_t row = (uint32_t)(q4 * 32 + lane);
    const uint32_t row_off = row * 128u, sw = row & 7u;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q4 * 32) << 16);
#pragma unroll
    for (int j = 0; j < COLS; j++) acc[j] = 0.f;
    int drained = 0;
    auto drain = [&]() {
      const int buf = drained % L::BUFS;
      ok = small_wait(smem_u32(&ss->seg_full[buf]), (uint32_t)((drained / L::BUFS) & 1), ss, p.status, 51);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        float v[16];
        tmem_ld16(t_lane + (uint32_t)(buf * TN + half * COLS + c), v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; j++) acc[c + j] += v[j];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_at(smem_u32(&ss->seg_empty[buf]));
      drained++;
    };
    pdl_grid_wait();   // (before the addend, the residual and the output are touched; the tiles come after it anyway)
    if (CS == 1 && p.shift && !RAGGED) {
#pragma unroll
      for (int j = 0; j < COLS; j += 4) {
        const int n = n0 + half * COLS + j;
        if (n >= p.N) break;
        const float4 b = pdl_ld(reinterpret_cast<const float4*>(p.shift + n));
        acc[j] = p.shift_mul * b.x;
        acc[j + 1] = p.shift_mul * b.y;
        acc[j + 2] = p.shift_mul * b.z;
        acc[j + 3] = p.shift_mul * b.w;
      }
    }
    const uint32_t full0 = smem_u32(&ss->full[0]), empty0 = smem_u32(&ss->empty[0]), tfull0 = smem_u32(&ss->t_full[0]);
    // stage and tensor-memory stage of K block kb; `old` = those of kb - T_ST, whose commit frees the latter
    int st = half, ts = half;
    uint32_t full_par = 0;
    for (int kb = half; kb < nkb && ok; kb += 2) {
      // the MMAs of a segment go into the accumulator of the segment BUFS before it
      const int seg = kb / SEG_KBLOCKS < nseg ? kb / SEG_KBLOCKS : nseg - 1;
      while (ok && seg >= drained + L::BUFS) drain();
      if (!ok) break;
      // K block kb - T_ST: its MMAs have read the part of tensor memory that this one's parts go to.  With an odd number of
      // stages they have also read this stage, which the other group waited for then: not before that may this group
      // wait for the stage's next phase, or it takes the end of the phase before the last for it.  (Loads arrive in any
      // order: block 1 there and block 0 not, and block 0's bytes were split as block 3's.)
      const int old = kb - L::T_ST;
      static_assert(L::STAGES % 2 == 0 || L::STAGES == L::T_ST, "a stage's phases are waited for one by one");
      auto wait_old = [&]() {
        return old < 0 || small_wait(empty0 + (uint32_t)(old % L::STAGES) * 8u, (uint32_t)((old / L::STAGES) & 1), ss, p.status, 53);
      };
      if (L::STAGES % 2) ok = wait_old();
      ok = ok && small_wait(full0 + (uint32_t)st * 8u, full_par, ss, p.status, 52);
      if (!ok) break;
      const unsigned char* src = smem + st * L::STAGE + row_off;
      const uint32_t dst = t_lane + (uint32_t)(L::A_COL0 + ts * 64);
      // (half a row at a time: the sums of the tile are live in registers too)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        float hi[16], lo[16];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const float4 x = *reinterpret_cast<const float4*>(src + (((uint32_t)(h * 4 + c) ^ sw) << 4));
          const float e[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int t = 0; t < 4; t++) {
            hi[c * 4 + t] = e[t];
            lo[c * 4 + t] = e[t] - __uint_as_float(__float_as_uint(e[t]) & 0xffffe000u);
          }
        }
        if (h == 0) {
          if (L::STAGES % 2 == 0) ok = wait_old();   // (with the first half of the row on its way)
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        tmem_st16(dst + (uint32_t)(h * 16), hi);
        if (!p.single_pass) tmem_st16(dst + 32u + (uint32_t)(h * 16), lo);
      }
      if (!ok) break;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_at(tfull0 + (uint32_t)ts * 8u);
      st += 2;
      if (st >= L::STAGES) { st -= L::STAGES; full_par ^= 1; }
      ts += 2;
      if (ts >= L::T_ST) ts -= L::T_ST;
    }
    while (ok && drained < nseg) drain();
  } else if (warp == SM_W_WARP) {
    // ============================================================================ weight tiles
    if (elect_one()) {
      const uint32_t w_bytes = (p.single_pass ? 1u : 2u) * (uint32_t)L::W_BYTES;
      // A constant weight whose split is known to be finished is no output of a grid still running: its first tiles
      // come in while the grids before this one finish.
      if (!w_early) pdl_grid_wait();
      const int tap0 = kb0 / p.cblocks;
      int cb = kb0 - tap0 * p.cblocks, kx0 = tap0 * p.ch_in + cb * BLOCK_K;   // a tap's last block may be short
      uint32_t bar = smem_u32(&ss->full[0]), dst = smem_u32(smem) + (uint32_t)A_TILE_BYTES, par = 1;
      constexpr uint32_t to_empty = (uint32_t)(offsetof(SmallShared, empty) - offsetof(SmallShared, full));
      const int row0 = p.w_row0 + n0;
      int st = 0, to_end = p.kblocks - kb0;
      for (int kb = 0; kb < nkb; kb++) {
        if (kb >= L::STAGES && !small_wait(bar + to_empty, par, ss, p.status, 54)) break;
        expect_at(bar, w_bytes);
        tma_load_2d_at(dst, &map_w_hi, bar, kx0, row0);
        if (!p.single_pass) tma_load_2d_at(dst + (uint32_t)L::W_BYTES, &map_w_lo, bar, kx0, row0);
        kx0 += BLOCK_K;
        if (++cb == p.cblocks) {
          cb = 0;
          kx0 += p.ch_in - p.cblocks * BLOCK_K;
        }
        if (--to_end == 0) cb = kx0 = 0;
        bar += 8u;
        dst += (uint32_t)L::STAGE;
        if (++st == L::STAGES) {
          st = 0;
          bar -= L::STAGES * 8u;
          dst -= (uint32_t)L::BYTES;
          par ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == SM_A_WARP) {
    // ============================================================================ A tiles
    if (elect_one()) {
      const uint32_t hw = (uint32_t)p.out_h * (uint32_t)p.out_w;
      const int64_t img = m0 / hw;
      const uint32_t rem = (uint32_t)(m0 - img * hw);
      const int oy = (int)(rem / (uint32_t)p.out_w), ox = (int)rem - oy * p.out_w;
      const int cw = ox * p.stride_w - p.pad_l, ch = oy * p.stride_h - p.pad_t;
      const int tap0 = kb0 / p.cblocks;
      int c0 = (kb0 - tap0 * p.cblocks) * BLOCK_K, ky = tap0 / p.k_w, kx = tap0 - ky * p.k_w;
      pdl_grid_wait();
      pdl_let_next_start();
      uint32_t bar = smem_u32(&ss->full[0]), dst = smem_u32(smem), par = 1;
      constexpr uint32_t to_empty = (uint32_t)(offsetof(SmallShared, empty) - offsetof(SmallShared, full));
      int st = 0, dx = kx * p.dil_w, dy = ky * p.dil_h, taps = p.k_h * p.k_w - tap0;
      for (int kb = 0; kb < nkb; kb++) {
        if (kb >= L::STAGES && !small_wait(bar + to_empty, par, ss, p.status, 55)) break;
        expect_at(bar, (uint32_t)A_TILE_BYTES);
        tma_load_im2col_at(dst, &map_a, bar, c0, cw, ch, (int)img, dx, dy);
        c0 += BLOCK_K;
        if (c0 >= p.ch_in) {
          c0 = 0;
          dx += p.dil_w;
          if (++kx == p.k_w) { kx = 0; dx = 0; dy += p.dil_h; }
          if (--taps == 0) kx = dx = dy = 0;
        }
        bar += 8u;
        dst += (uint32_t)L::STAGE;
        if (++st == L::STAGES) {
          st = 0;
          bar -= L::STAGES * 8u;
          dst -= (uint32_t)L::BYTES;
          par ^= 1;
        }
      }
    }
    __syncwarp();
  } else {
    // ============================================================================ MMA issuer
    const uint32_t leader = elect_one() ? 1u : 0u;
    const uint32_t idesc = make_idesc(TN);
    const uint64_t desc0 = make_smem_desc(smem_u32(smem) + (uint32_t)A_TILE_BYTES);
    const uint32_t top = (uint32_t)(desc0 >> 32), w0 = (uint32_t)desc0;
    const uint32_t tfull0 = smem_u32(&ss->t_full[0]), empty0 = smem_u32(&ss->empty[0]);
    uint32_t wh = w0, a_hi = tmem_base + (uint32_t)L::A_COL0, t_bar = tfull0, e_bar = empty0, t_par = 0;
    int st = 0, ts = 0, left = nkb;
    bool tok = false, go = true;
    for (int seg = 0; seg < nseg && go; seg++) {
      const int n = seg == nseg - 1 ? left : SEG_KBLOCKS, buf = seg % L::BUFS;
      if (seg >= L::BUFS)
        go = small_wait(smem_u32(&ss->seg_empty[buf]), (uint32_t)((seg / L::BUFS) & 1) ^ 1, ss, p.status, 56);
      const uint32_t d = tmem_base + (uint32_t)(buf * TN);
      for (int i = 0; i < n && go; i++) {
        // (the splitters have seen the stage full, W included)
        if (!tok) go = small_wait(t_bar, t_par, ss, p.status, 57);
        if (!go) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_lo = a_hi + 32u, wl = wh + (uint32_t)(L::W_BYTES >> 4), first = i ? 1u : 0u;
        const uint32_t t_bar_n = ts + 1 == L::T_ST ? tfull0 : t_bar + 8u, t_par_n = ts + 1 == L::T_ST ? t_par ^ 1 : t_par;
        left--;
        if (p.single_pass) {
#pragma unroll
          for (int k = 0; k < BLOCK_K / 8; k++)
            umma_by(leader, d, a_hi + (uint32_t)(k * 8), wh + (uint32_t)(k * 2), top, idesc, k ? 1u : first);
          tok = left > 0 && test_at(t_bar_n, t_par_n);
        } else {
#pragma unroll
          for (int k = 0; k < BLOCK_K / 8; k++) {
            const uint32_t adv = (uint32_t)(k * 2), acol = (uint32_t)(k * 8);
            umma_by(leader, d, a_lo + acol, wh + adv, top, idesc, k ? 1u : first);
            umma_by(leader, d, a_hi + acol, wl + adv, top, idesc, 1u);
            umma_by(leader, d, a_hi + acol, wh + adv, top, idesc, 1u);
            // ask for the next stage with MMAs of this one queued (see PROBE_AFTER_K)
            if (k == PROBE_AFTER_K) tok = left > 0 && test_at(t_bar_n, t_par_n);
          }
        }
        commit_by(leader, e_bar);
        t_bar = t_bar_n;
        t_par = t_par_n;
        a_hi += 64u;
        if (++ts == L::T_ST) { ts = 0; a_hi -= 64u * L::T_ST; }
        wh += (uint32_t)(L::STAGE >> 4);
        e_bar += 8u;
        if (++st == L::STAGES) { st = 0; wh = w0; e_bar = empty0; }
      }
      commit_by(leader, smem_u32(&ss->seg_full[buf]));
    }
    __syncwarp();
  }

  // ------------------------------------------------------------------------------------ exchange
  if (CS > 1 && threadIdx.x == 0) expect_at(smem_u32(&ss->recv), (uint32_t)(mine * CS * TN * 4));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (CS > 1) {
    if (!L::OWN_EXCHANGE)   // the stages are free in every CTA of the cluster behind this barrier
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (CS == 1 || L::OWN_EXCHANGE) __syncthreads();   // tensor memory has been read
  if (warp == SM_MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SM_TMEM_COLS));
  }
  if (warp >= SM_SPLIT_WARPS) {
    if (ss->abort_flag == 0) return;
  } else {
    const uint32_t row = (uint32_t)(q4 * 32 + lane);
    const bool sums_ok = ok && ss->abort_flag == 0;
    const uint32_t base = smem_u32(smem) + (uint32_t)L::EXCHANGE_OFF;
    if (CS > 1) {
      if (sums_ok && (int)row < rows) {
        const uint32_t peer = row / (uint32_t)share, drow = row - peer * (uint32_t)share;
        const uint32_t dst = map_to_rank(base + (uint32_t)(rank * CELLS * ROWS) * 16u, peer);
        const uint32_t bar = map_to_rank(smem_u32(&ss->recv), peer);
#pragma unroll
        for (int c = 0; c < COLS / 4; c++) {
          const uint32_t cell = (uint32_t)(half * (COLS / 4) + c);
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                           dst + exchange_slot<ROWS>(drow, cell) * 16u),
                       "f"(acc[c * 4]), "f"(acc[c * 4 + 1]), "f"(acc[c * 4 + 2]), "f"(acc[c * 4 + 3]), "r"(bar)
                       : "memory");
        }
      }
    } else if (sums_ok) {
#pragma unroll
      for (int c = 0; c < COLS / 4; c++) {
        const uint32_t cell = (uint32_t)(half * (COLS / 4) + c);
        *reinterpret_cast<float4*>(smem + L::EXCHANGE_OFF + exchange_slot<ROWS>(row, cell) * 16u) =
            make_float4(acc[c * 4], acc[c * 4 + 1], acc[c * 4 + 2], acc[c * 4 + 3]);
      }
    }
    // residual and addend are on their way while the sums are
    float4 out[ITEMS], res[ITEMS];   // out: the addend, in front of the sums or (rows of any length) behind them
    bool live[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      const int item = threadIdx.x + i * SM_EPI_THREADS, r = item / CELLS, n = n0 + (item % CELLS) * 4;
      const int64_t m = m0 + rank * share + r;
      live[i] = r < mine && n < p.N;
      out[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live[i]) {
        if ((CS > 1 || RAGGED) && p.shift) {
          const float4 b = small_cell<RAGGED>(p.shift + n, n, p.N);
          out[i] = RAGGED ? make_float4(__fmul_rn(p.shift_mul, b.x), __fmul_rn(p.shift_mul, b.y), __fmul_rn(p.shift_mul, b.z), __fmul_rn(p.shift_mul, b.w))
                          : make_float4(p.shift_mul * b.x, p.shift_mul * b.y, p.shift_mul * b.z, p.shift_mul * b.w);
        }
        if (p.residual) res[i] = small_cell<RAGGED>(p.residual + m * p.res_stride + n, n, p.N);
      }
    }
    if (CS > 1) ok = sums_ok && small_wait(smem_u32(&ss->recv), 0, ss, p.status, 59);
    else {
      asm volatile("bar.sync 1, %0;" ::"n"(SM_EPI_THREADS) : "memory");
      ok = sums_ok;
    }
    if (ok) {
#pragma unroll
      for (int i = 0; i < ITEMS; i++) {
        if (!live[i]) continue;
        const int item = threadIdx.x + i * SM_EPI_THREADS, r = item / CELLS, cell = item % CELLS;
        const unsigned char* src = smem + L::EXCHANGE_OFF + exchange_slot<ROWS>((uint32_t)r, (uint32_t)cell) * 16u;
        float4 s = CS == 1 ? *reinterpret_cast<const float4*>(src) : RAGGED ? make_float4(0.f, 0.f, 0.f, 0.f) : out[i];
#pragma unroll
        for (int q = 0; CS > 1 && q < CS; q++) {
          const float4 v = *reinterpret_cast<const float4*>(src + q * (CELLS * ROWS * 16));
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (RAGGED) {
          s.x += out[i].x; s.y += out[i].y; s.z += out[i].z; s.w += out[i].w;
        }
        if (p.residual) {
          s.x = fmaf(p.res_mul, res[i].x, s.x);
          s.y = fmaf(p.res_mul, res[i].y, s.y);
          s.z = fmaf(p.res_mul, res[i].z, s.z);
          s.w = fmaf(p.res_mul, res[i].w, s.w);
        }
        if (p.relu) {
          s.x = relu_nan(s.x); s.y = relu_nan(s.y); s.z = relu_nan(s.z); s.w = relu_nan(s.w);
        }
        float* dst = y + (m0 + rank * share + r) * p.y_stride + n0 + cell * 4;
        if (!RAGGED) {
          *reinterpret_cast<float4*>(dst) = s;
        } else {
          const int left = p.N - n0 - cell * 4;
          dst[0] = s.x;
          if (left > 1) dst[1] = s.y;
          if (left > 2) dst[2] = s.z;
          if (left > 3) dst[3] = s.w;
        }
      }
    }
  }
  // A wait ran out: stay until the cluster's other CTAs have given up as well (their sums must find this CTA's memory).
  if (CS > 1 && (ss->abort_flag || !ok)) {
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 2 * WAIT_LIMIT_NS) __nanosleep(1000000);
  }
}
