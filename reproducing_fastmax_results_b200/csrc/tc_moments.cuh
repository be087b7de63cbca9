// Moment states alone: S = Phi(X)^T Y over all tokens (state-only calls: X = k, Y = [v | 1]; gradient moments: X = q,
// Y = dO').  Included by tc_kernels.cu inside fm::tc.
//
// Without an output there is no order between the chunks, so the tokens of a head may be cut over several thread blocks and
// no copy of the state is needed.  A block takes up to four feature tiles (the accumulators) of one head and a range of
// 128-token chunks.  Two groups of eight producer warps form the slabs (a tile's features of a chunk) in turn, in registers, and
// store them to tensor memory as the A operand; thread = feature, tokens from the transposed copy.  The row of the feature's
// first factor is kept in registers across a group's tiles that share it.
// TMEM: four 80-column accumulators, three 64-column slots.
//
// No unit is full: 8 heads of 32768 x 64 keep the shared-memory pipe busy for 52 % of the clocks, the tensor pipe for 36 %, the
// schedulers for 39 %.  One product of 80 columns per K step instead of one of 64 and one of 16, and slabs in turn instead of every
// warp at every slab (half as many hand-overs): 72.6 -> 69.6 us for 64 heads of 1999 x 64, 578 -> 572 for the segments of 8 heads of
// 131072; 128 heads of one chunk, whose slabs have nothing beside them, 39.2 -> 41.4.
#pragma once

namespace mo {

constexpr int THREADS = 576;
constexpr int W_MMA = 16, W_TMA = 17;
constexpr int STAGES = 4;
// D: head dim.  Feature tiles: two 64-row pair units each, the last one holds the linear and constant rows.
template <int D>
struct Lay {
  static constexpr int NB = D / 8;
  static constexpr int PAIR_TILES = NB * (NB + 1) / 4;
  static constexpr int TILES = PAIR_TILES + 1;
  static constexpr int KT_BOX = D * s2::KT_ROW;           // D dims x 72 tokens
  // Y and its tail (ones or -delta, then zeros): 128 tokens, 128-byte swizzled rows, one 64-column group behind the other
  static constexpr int OFF_T = REGION, OFF_XT = 2 * REGION, STAGE = (OFF_XT + 2 * KT_BOX + 1023) / 1024 * 1024;
  static constexpr int OFF_BAR = STAGES * STAGE;
  static constexpr int SMEM_BYTES = OFF_BAR + 512 + 1024;
  static constexpr int LD = D + 4;
  static_assert((NB * (NB + 1) / 2) % 2 == 0, "whole tiles of two pair units");
  static_assert(KT_BOX % 128 == 0, "TMA destinations");
  static_assert(4 * CH * LD * 4 <= STAGES * STAGE, "the output rows are staged over the tiles");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};
constexpr int B_FULL = 0, B_EMPTY = STAGES, B_SLOT = 2 * STAGES, B_FREE = B_SLOT + 3, B_DONE = B_FREE + 6, B_COUNT = B_DONE + 1;
constexpr int NC = 80;            // accumulator columns of a tile: 64 of Y (narrow heads: zeros behind them), the tail, zeros
constexpr uint32_t COL_A = 4 * NC;

struct Params {
  float* out;          // [BH][state_rows][D + 4]; per_split: [BH][nsplit][state_rows][D + 4]
  int n;               // tokens
  int bh, heads, nchunks, chunks_per_split, nsplit;
  int nslices, tps, tile_first, state_rows;
  int dop;             // Y is dO' and its tail column comes from memory (column D); else the tail is ones
  int per_split;       // every split has a state of its own
  int add;             // add to `out` instead of storing
};

template <int D>
__global__ void __launch_bounds__(THREADS, 1)
moments_kernel(const __grid_constant__ CUtensorMap tmxt, const __grid_constant__ CUtensorMap tmy, const __grid_constant__ CUtensorMap tmt,
               const Params P) {
  using L = Lay<D>;
  constexpr int STAGE = L::STAGE, OFF_XT = L::OFF_XT, OFF_BAR = L::OFF_BAR, KT_BOX = L::KT_BOX, LIN = L::TILES - 1;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // slice-major: the last slice of a head may have fewer tiles, and these shorter blocks end the grid
  const int units = P.bh * P.nsplit, slice = blockIdx.x / units, rest = blockIdx.x - slice * units;
  const int head = rest / P.nsplit, split = rest - head * P.nsplit;
  const int b_idx = head / P.heads, h_idx = head - b_idx * P.heads;
  const int tile0 = P.tile_first + slice * P.tps;
  const int ntl = min(P.tps, L::TILES - tile0);
  const int c0 = split * P.chunks_per_split, c1 = min(P.nchunks, c0 + P.chunks_per_split);
  const int nc = c1 - c0;

  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) mbar_init(&bars[i], (i >= B_SLOT && i < B_FREE) ? 8 : 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (!P.dop)   // the tail of [v | 1], the same in every stage (features of tokens past the last one are zero)
    for (int i = tid; i < STAGES * CH * 8; i += THREADS) {
      const int row = (i >> 3) % CH;
      *reinterpret_cast<uint4*>(sm + i / (8 * CH) * STAGE + L::OFF_T + row * 128 + (i & 7) * 16) = make_uint4((i & 7) == (row & 7) ? 0x00003F80u : 0u, 0u, 0u, 0u);
    }
  fence_proxy_async_smem();
  if (w == W_MMA) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto WAIT = [&](int bar, uint32_t phase, int code) {
    if (!mbar_try_wait(&bars[bar], phase & 1u) && *abort_flag == 0 && !s2::wait_slow(&bars[bar], phase & 1u, abort_flag)) s2::fail_record(code, abort_flag);
  };

  int loaded = 0;
  if (w == W_TMA) {
    for (int i = 0; i < nc; ++i) {
      const int s = i % STAGES;
      if (i >= STAGES) WAIT(B_EMPTY + s, (uint32_t)(i / STAGES) - 1u, 110);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        uint8_t* st = sm + s * STAGE;
        const int tok = (c0 + i) * CH;
        mbar_arrive_expect_tx(&bars[B_FULL + s], 2 * KT_BOX + (P.dop ? 2 : 1) * REGION);
        tma_load_4d(st, &tmy, &bars[B_FULL + s], 0, tok, h_idx, b_idx);
        if (P.dop) tma_load_4d(st + L::OFF_T, &tmt, &bars[B_FULL + s], D, tok, h_idx, b_idx);
        tma_load_3d(st + OFF_XT, &tmxt, &bars[B_FULL + s], tok, 0, head);
        tma_load_3d(st + OFF_XT + KT_BOX, &tmxt, &bars[B_FULL + s], tok + 64, 0, head);
      }
      loaded = i + 1;
    }
  } else if (w == W_MMA) {
    constexpr uint32_t ID = make_idesc_bf16(128, NC, 0, 1);
    const uint64_t dY = make_smem_desc(smem_u32(sm), L::OFF_T, 1024, 2);
    uint32_t k = 0;   // slabs so far
    for (int i = 0; i < nc; ++i) {
      const uint32_t s = (uint32_t)i % STAGES;
      WAIT(B_FULL + (int)s, (uint32_t)(i / STAGES), 111);
      for (int t = 0; t < ntl; ++t, ++k) {
        const uint32_t slot = k % 3u;
        WAIT(B_SLOT + (int)slot, k / 3u, 112);
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          mma_ts_elect(tmem + NC * t, tmem + COL_A + 64u * slot + 8u * kk, dY + (uint64_t)(s * (STAGE >> 4) + 128 * kk), ID, (i > 0 || kk > 0) ? 1u : 0u);
        mma_commit_elect(&bars[B_FREE + (k + 3u) % 6u]);   // to the group that fills the slot next
      }
      mma_commit_elect(&bars[B_EMPTY + s]);
    }
    mma_commit_elect(&bars[B_DONE]);
    mbar_wait_bounded(&bars[B_DONE], 0, WAIT_CYCLES);   // (also after a failure: leave only after the products in flight)
  } else {
    const uint32_t group = (uint32_t)w >> 3;            // slabs take turns between the two groups
    const int half = (w >> 2) & 1, row = (w & 3) * 32 + lane;   // 64 tokens of the chunk; feature row of a tile
    const uint32_t lane_addr = tmem + ((uint32_t)((w & 3) * 32) << 16);
    // byte offsets of the two factor rows of each tile's feature (16 bits each); b0 < 0: the linear tile
    const int f = row & 63;
    uint32_t rows[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      int a = 0, b = 0;
      if (t < ntl && tile0 + t < LIN) pair_decode(2 * (tile0 + t) + (row >> 6), L::NB, a, b);   // warp-uniform
      rows[t] = (uint32_t)((8 * a + (f >> 3)) * s2::KT_ROW) | (uint32_t)((8 * b + (f & 7)) * s2::KT_ROW) << 16;
      if (tile0 + t == LIN) rows[t] = (uint32_t)((f & (D - 1)) * s2::KT_ROW) | (uint32_t)((f & (D - 1)) * s2::KT_ROW) << 16;
    }
    uint32_t k = 0;   // slabs so far, of both groups
    for (int i = 0; i < nc; ++i) {
      const int s = i % STAGES;
      const uint8_t* box = sm + s * STAGE + OFF_XT + half * KT_BOX;
      auto load = [&](uint4 (&x)[8], uint32_t off) {
        const uint4* p = reinterpret_cast<const uint4*>(box + off);
#pragma unroll
        for (int c = 0; c < 8; ++c) x[c] = p[c];
      };
      uint4 xa[8];
      uint32_t have = ~0u;   // the row in xa
#pragma unroll
      for (int t = 0; t < 4; ++t, ++k) {
        if (t >= ntl) break;
        if ((k & 1u) != group) continue;
        // (a group without a slab in this chunk does not wait for it: the stage may be filled again before it would look)
        if (t < 2) WAIT(B_FULL + s, (uint32_t)(i / STAGES), 113);
        uint32_t r[32];
        {
          uint4 xb[8];
          load(xb, rows[t] >> 16);
#pragma unroll
          for (int c = 0; c < 8; ++c) { r[4 * c] = xb[c].x; r[4 * c + 1] = xb[c].y; r[4 * c + 2] = xb[c].z; r[4 * c + 3] = xb[c].w; }
        }
        if (tile0 + t < LIN) {
          if ((rows[t] & 0xffffu) != have) {
            have = rows[t] & 0xffffu;
            load(xa, have);
          }
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            r[4 * c] = hmul2_u32(xa[c].x, r[4 * c]);
            r[4 * c + 1] = hmul2_u32(xa[c].y, r[4 * c + 1]);
            r[4 * c + 2] = hmul2_u32(xa[c].z, r[4 * c + 2]);
            r[4 * c + 3] = hmul2_u32(xa[c].w, r[4 * c + 3]);
          }
        } else if (row >= D) {   // the constant feature (row D), zero for tokens past the last one, and nothing
          const int left = row == D ? P.n - ((c0 + i) * CH + 64 * half) : 0;
#pragma unroll
          for (int c = 0; c < 32; ++c) r[c] = (2 * c < left ? 0x00003F80u : 0u) | (2 * c + 1 < left ? 0x3F800000u : 0u);
        }
        const uint32_t slot = k % 3u;
        if (k >= 3) WAIT(B_FREE + (int)(k % 6u), k / 6u - (k % 6u < 3u ? 1u : 0u), 114);
        tc_fence_after_sync();
        tmem_st32(lane_addr + COL_A + 64u * slot + 32u * half, r);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[B_SLOT + slot]);
      }
    }
    WAIT(B_DONE, 0, 115);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort_flag == 0) {
    // accumulators -> staging rows of D + 4 floats -> the state's rows, which lie one behind the other; producer group g: tile g
    const int g = w >> 2;
    if (g < ntl) {
      float* stage = reinterpret_cast<float*>(sm) + g * CH * L::LD;
      const int row = (w & 3) * 32 + lane;
      const uint32_t a = tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)(NC * g);
      float4* dst = reinterpret_cast<float4*>(stage + row * L::LD);
      uint32_t r[32], r8[8];
      tmem_ld8(a + 64u, r8);
#pragma unroll
      for (int half = 0; half < D / 32; ++half) {
        tmem_ld32(a + 32u * half, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          dst[8 * half + j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
      }
      dst[D / 4] = make_float4(__uint_as_float(r8[0]), 0.f, 0.f, 0.f);
      fence_proxy_async_smem();
      named_bar_sync(1 + g, 128);
      if ((w & 3) == 0 && lane == 0) {
        const int row0 = (tile0 + g - P.tile_first) * CH, rows = min(CH, P.state_rows - row0);
        float* out = P.out + ((long long)(P.per_split ? head * P.nsplit + split : head) * P.state_rows + row0) * L::LD;
        if (P.add) bulk_reduce_add_f32(out, stage, (uint32_t)(rows * L::LD * 4));
        else bulk_store(out, stage, (uint32_t)(rows * L::LD * 4));
        bulk_commit_group();
        bulk_wait_read_all();
      }
    }
  } else if (w == W_TMA) {
    for (int i = loaded > STAGES ? loaded - STAGES : 0; i < loaded; ++i)
      mbar_wait_bounded(&bars[B_FULL + i % STAGES], (uint32_t)(i / STAGES) & 1u, WAIT_CYCLES);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (w == W_MMA) tmem_dealloc(tmem, 512);
}

}  // namespace mo
