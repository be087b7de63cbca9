// Moment states alone: S = Phi(X)^T Y over all tokens (state-only calls: X = k, Y = [v | 1]; gradient moments: X = q,
// Y = dO').  Included by tc_kernels.cu inside fm::tc.
//
// Without an output there is no order between the chunks, so the tokens of a head may be cut over several thread blocks and
// no copy of the state is needed.  A block takes up to four feature tiles (the accumulators) of one head and a range of
// 128-token chunks.  Four producer warpgroups, one per 32-token quarter of a chunk, form the products in registers and store
// them to tensor memory as the A operand; thread = feature, tokens from the transposed copy.  The row of the feature's first
// factor is kept in registers across the tiles that share it: 1.25 rows read per feature instead of two (a 128-bit load of a
// warp takes four wavefronts whatever its lanes share).
// TMEM: four 80-column accumulators, three 64-column slots.
//
// 620 clocks per tile and chunk.  No unit is full: 64 heads of 4096 x 64 (130 us) keep the shared-memory pipe busy for 58 % of the
// time, the tensor pipe for 43 % (two products per K step, N = D and N = 16), the schedulers for 48 %.
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
  static constexpr int NC = D + 16;                       // accumulator columns of a tile: Y and its tail column
  static constexpr int KT_BOX = D * s2::KT_ROW;           // D dims x 72 tokens
  // Y: 128 tokens, 128-byte swizzled rows; tail (-delta of dO'): one 8-column block (8 columns used as 16: zeros follow)
  static constexpr int OFF_T = REGION, OFF_XT = REGION + BLK, STAGE = (OFF_XT + 2 * KT_BOX + 1023) / 1024 * 1024;
  static constexpr int OFF_ONES = STAGES * STAGE;         // the tail of [v | 1]: one constant block of ones, then a block of zeros
  static constexpr int OFF_BAR = OFF_ONES + 2 * BLK;
  static constexpr int SMEM_BYTES = OFF_BAR + 512 + 1024;
  static constexpr int LD = D + 4;
  static_assert((NB * (NB + 1) / 2) % 2 == 0, "whole tiles of two pair units");
  static_assert(KT_BOX % 128 == 0, "TMA destinations");
  static_assert(4 * CH * LD * 4 <= STAGES * STAGE, "the output rows are staged over the tiles");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};
constexpr int B_FULL = 0, B_EMPTY = STAGES, B_SLOT = 2 * STAGES, B_FREE = B_SLOT + 3, B_DONE = B_FREE + 3, B_COUNT = B_DONE + 1;
constexpr uint32_t COL_A = 320;   // behind four accumulators of 80 columns

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
    for (int i = 0; i < B_COUNT; ++i) mbar_init(&bars[i], (i >= B_SLOT && i < B_FREE) ? 16 : 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  for (int i = tid; i < 2 * CH; i += THREADS)   // (features of tokens past the last one are zero)
    *reinterpret_cast<uint4*>(sm + L::OFF_ONES + i * 16) = make_uint4(i < CH ? 0x00003F80u : 0u, 0u, 0u, 0u);
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
        mbar_arrive_expect_tx(&bars[B_FULL + s], 2 * KT_BOX + REGION + (P.dop ? BLK : 0));
        tma_load_4d(st, &tmy, &bars[B_FULL + s], 0, tok, h_idx, b_idx);
        if (P.dop) tma_load_4d(st + L::OFF_T, &tmt, &bars[B_FULL + s], D, tok, h_idx, b_idx);
        tma_load_3d(st + OFF_XT, &tmxt, &bars[B_FULL + s], tok, 0, head);
        tma_load_3d(st + OFF_XT + KT_BOX, &tmxt, &bars[B_FULL + s], tok + 64, 0, head);
      }
      loaded = i + 1;
    }
  } else if (w == W_MMA) {
    constexpr uint32_t ID = make_idesc_bf16(128, D, 0, 1), ID_T = make_idesc_bf16(128, 16, 0, 1);
    const uint64_t dY = make_smem_desc(smem_u32(sm), REGION, 1024, 2);
    const uint32_t zeros = smem_u32(sm + L::OFF_ONES + BLK);
    uint32_t k = 0;   // slabs so far
    for (int i = 0; i < nc; ++i) {
      const uint32_t s = (uint32_t)i % STAGES;
      WAIT(B_FULL + (int)s, (uint32_t)(i / STAGES), 111);
      // tail operand: its block of eight columns, and the zeros a fixed distance behind it
      const uint32_t tail = P.dop ? smem_u32(sm + s * STAGE + L::OFF_T) : smem_u32(sm + L::OFF_ONES);
      const uint64_t dT = make_smem_desc(tail, 128, zeros - tail, 0);
      for (int t = 0; t < ntl; ++t, ++k) {
        const uint32_t slot = k % 3u;
        WAIT(B_SLOT + (int)slot, k / 3u, 112);
        tc_fence_after_sync();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t a = tmem + COL_A + 64u * slot + 8u * kk, acc = (i > 0 || kk > 0) ? 1u : 0u;
          mma_ts_elect(tmem + L::NC * t, a, dY + (uint64_t)(s * (STAGE >> 4) + 128 * kk), ID, acc);
          mma_ts_elect(tmem + L::NC * t + D, a, dT + (uint64_t)(16 * kk), ID_T, acc);
        }
        mma_commit_elect(&bars[B_FREE + slot]);
      }
      mma_commit_elect(&bars[B_EMPTY + s]);
    }
    mma_commit_elect(&bars[B_DONE]);
    mbar_wait_bounded(&bars[B_DONE], 0, WAIT_CYCLES);   // (also after a failure: leave only after the products in flight)
  } else {
    const int g = w >> 2, row = (w & 3) * 32 + lane;    // producer group = quarter of the chunk; feature row of a tile
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
    uint32_t k = 0;
    for (int i = 0; i < nc; ++i) {
      const int s = i % STAGES;
      WAIT(B_FULL + s, (uint32_t)(i / STAGES), 113);
      const uint8_t* box = sm + s * STAGE + OFF_XT + (g >> 1) * KT_BOX + (g & 1) * 64;
      uint4 xa[4], xb[4];
      auto load = [&](uint4 (&x)[4], uint32_t off) {
        const uint4* p = reinterpret_cast<const uint4*>(box + off);
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = p[c];
      };
      load(xb, rows[0] >> 16);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t < ntl) {
          uint32_t r[16];
          if (tile0 + t < LIN) {
            if (t == 0 || (rows[t] & 0xffffu) != (rows[t > 0 ? t - 1 : 0] & 0xffffu)) load(xa, rows[t] & 0xffffu);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              r[4 * c] = hmul2_u32(xa[c].x, xb[c].x);
              r[4 * c + 1] = hmul2_u32(xa[c].y, xb[c].y);
              r[4 * c + 2] = hmul2_u32(xa[c].z, xb[c].z);
              r[4 * c + 3] = hmul2_u32(xa[c].w, xb[c].w);
            }
          } else if (row < D) {
#pragma unroll
            for (int c = 0; c < 4; ++c) { r[4 * c] = xb[c].x; r[4 * c + 1] = xb[c].y; r[4 * c + 2] = xb[c].z; r[4 * c + 3] = xb[c].w; }
          } else {   // the constant feature (row D), zero for tokens past the last one, and nothing
            const int left = row == D ? P.n - ((c0 + i) * CH + 32 * g) : 0;
#pragma unroll
            for (int c = 0; c < 16; ++c) r[c] = (2 * c < left ? 0x00003F80u : 0u) | (2 * c + 1 < left ? 0x3F800000u : 0u);
          }
          if (t + 1 < ntl) load(xb, rows[t < 3 ? t + 1 : 3] >> 16);   // in flight while this slab is handed over
          const uint32_t slot = k % 3u;
          if (k >= 3) WAIT(B_FREE + (int)slot, k / 3u - 1u, 114);
          tc_fence_after_sync();
          tmem_st16(lane_addr + COL_A + 64u * slot + 16u * g, r);
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[B_SLOT + slot]);
          ++k;
        }
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
      const uint32_t a = tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)(L::NC * g);
      float4* dst = reinterpret_cast<float4*>(stage + row * L::LD);
      uint32_t r[32], r8[8];
      tmem_ld8(a + (uint32_t)D, r8);
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
