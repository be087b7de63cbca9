// Long float32 sequences, head dim 32: windows of pairs and moment states as in long_kernels.cuh, at float32 accuracy.  Included
// by pair_kernels.cu inside fm::lng.
//
// Products are sums of six bf16 piece products (see pair_f32.cuh).  The features are formed and split into their three pieces in
// registers, in float32 from the tensors themselves; states are split once, when they are packed.  The tensor pipe adds with
// truncation, so an accumulator lives for one unit (64 features, or 64 tokens of a moment) and the drain warps add it to
// float32 totals in registers.  What bounds all three kernels is starting products: 24 MMAs (13 in the chain) of N = 48 per 64
// features and tile, one every 33 clocks, each 24 clocks of the tensor pipe, which is active in 48 % (apply) and 62 % (chain) of
// the clocks (ncu, 8 heads of 32768).  Measured, 8 heads x 131072 tokens, order 2: moments 419 us, packing 128, apply 370, chain 293; forward and
// backward with the pairwise windows 4.5 ms, where the CUDA-core engine (multiply-adds bound by its shared-memory reads, a scan
// over segments) took 22.5.
#pragma once

namespace f32 {

using pair::f32::split3;
constexpr int D = 32, NB = 4, NPAIR = 10, UNITS = 11;
constexpr int NC = 48;                        // columns: values, denominator, zeros
constexpr int PIECE = (NC / 8) * 1024;        // [block][64 rows][8 columns] bf16
constexpr int UNIT = 3 * PIECE;
constexpr int CST = 40, LD = 36;              // constant row of a state; row of an unpacked state
constexpr int CHUNK = 64;                     // tokens of a moment product
constexpr int SLOTS = 3, ACCS = 4;            // TMEM rings: A operands of 3 x 32 columns, accumulators of 48
constexpr uint32_t COL_SLOT = ACCS * NC;

// acc = sum over the piece products of A (TMEM, `pa` columns per piece) and B (shared memory), the smallest first
template <int KK>
__device__ __forceinline__ void product(uint32_t acc, uint32_t a, uint32_t pa, uint64_t b, uint32_t pb, uint32_t bk, uint32_t id, int kk_used) {
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    constexpr uint32_t PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
    for (int kk = 0; kk < KK; ++kk)
      if (kk < kk_used) mma_ts_elect(acc, a + pa * PA[t] + 8u * kk, b + (uint64_t)(pb * PB[t] + bk * kk), id, t > 0 || kk > 0);
  }
}
// adds 32 values and the denominator of an accumulator to a row's totals, and gives it back
__device__ __forceinline__ void drain(uint64_t (&tot)[17], uint32_t acc, uint64_t* free_bar, int lane) {
  uint32_t r[32], r8[8];
  tmem_ld32(acc, r);
  tmem_ld8(acc + 32u, r8);
  tmem_ld_wait();
  tc_fence_before_sync();
  __syncwarp();
  if (lane == 0) mbar_arrive(free_bar);
#pragma unroll
  for (int j = 0; j < 16; ++j) tot[j] = add2(tot[j], pack2u(r[2 * j], r[2 * j + 1]));
  tot[16] = add2(tot[16], pack2u(r8[0], 0u));
}

// ---- moments: raw state of every segment, [head][segment][rows][LD] = Phi(X)^T [Y | tail] ----------------------------------
// An item is two tiles of 128 features of one segment.  Producers: thread = feature, the two warpgroups take 32 tokens of each
// chunk; all lanes of a warp read the same token's row, so the reads are without conflicts and no transposed copy is needed.
namespace mo {
constexpr int THREADS = 512, W_MMA = 0, W_LOAD = 1, W_DRAIN = 4, W_PROD = 8;
constexpr int TILES = 6, LIN = 5;             // the last tile: 32 linear features and the constant one
constexpr int STAGES = 5, XB = CHUNK * 128, YB = CHUNK * 128, STAGE = XB + 3 * YB;
constexpr int OFF_OUT = STAGES * STAGE, OFF_BAR = OFF_OUT + 2 * 128 * LD * 4, BYTES = OFF_BAR + 512 + 1024;
static_assert(BYTES <= 232448, "shared memory budget");
constexpr int B_FULL = 0, B_EMPTY = B_FULL + STAGES, B_SLOT = B_EMPTY + STAGES, B_SLFREE = B_SLOT + SLOTS, B_ACC = B_SLFREE + SLOTS, B_AFREE = B_ACC + ACCS,
              B_DRAIN = B_AFREE + ACCS, B_COUNT = B_DRAIN + 1;

struct Params {
  float* out;
  int n, heads, seg, nsplit, nslices, nitems, tile_first, state_rows;
};
struct Maps {
  CUtensorMap x;   // float32 tensor, 64-row boxes of 32 columns, not swizzled
  CUtensorMap y;   // pieces with NC columns, 64-row boxes, swizzled
};
struct Item {
  int head, split, tile0, ntl, tok, nc;
};
__device__ __forceinline__ Item item(int idx, const Params& P) {   // slices of one segment side by side: they read the same chunks
  Item it;
  const int rest = idx / P.nslices;
  it.tile0 = P.tile_first + 2 * (idx - rest * P.nslices);
  it.ntl = min(2, TILES - it.tile0);
  it.head = rest / P.nsplit;
  it.split = rest - it.head * P.nsplit;
  it.tok = it.split * P.seg;
  it.nc = (min(P.n - it.tok, P.seg) + CHUNK - 1) / CHUNK;
  return it;
}

__global__ void __launch_bounds__(THREADS, 1) moments_kernel(const __grid_constant__ Maps M, const Params P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      uint32_t n = 1;
      if (i >= B_SLOT && i < B_SLFREE) n = 8;
      if (i >= B_AFREE && i < B_DRAIN) n = 4;
      mbar_init(&bars[i], n);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (w == W_MMA) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto WAIT = [&](int bar, uint32_t phase, int code) { wait_fast(&bars[bar], phase & 1u, code, abort_flag); };

  int loaded = 0;
  if (w == W_LOAD) {
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x) {
      const Item it = item(idx, P);
      const int b = it.head / P.heads, h = it.head - b * P.heads;
      for (int c = 0; c < it.nc; ++c) {
        const int s = loaded % STAGES;
        if (loaded >= STAGES) WAIT(B_EMPTY + s, (uint32_t)(loaded / STAGES) - 1u, 141);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          uint8_t* st = sm + s * STAGE;
          const int tok = it.tok + c * CHUNK;
          mbar_arrive_expect_tx(&bars[B_FULL + s], STAGE);
          tma_load_4d(st, &M.x, &bars[B_FULL + s], 0, tok, h, b);
          for (int p = 0; p < 3; ++p) tma_load_4d(st + XB + p * YB, &M.y, &bars[B_FULL + s], 0, tok, it.head, p);
        }
        ++loaded;
      }
    }
  } else if (w == W_MMA) {
    constexpr uint32_t ID = make_idesc_bf16(128, NC, 0, 1);
    const uint64_t dY = make_smem_desc(smem_u32(sm + XB), YB, 1024, 2);
    uint32_t seq = 0, k = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x) {
      const Item it = item(idx, P);
      for (int c = 0; c < it.nc; ++c, ++k) {
        const uint32_t s = k % STAGES;
        WAIT(B_FULL + (int)s, k / STAGES, 142);
        for (int t = 0; t < it.ntl; ++t, ++seq) {
          const uint32_t slot = seq % SLOTS, ab = seq % ACCS;
          WAIT(B_SLOT + (int)slot, seq / SLOTS, 143);
          if (seq >= ACCS) WAIT(B_AFREE + (int)ab, seq / ACCS - 1u, 144);
          tc_fence_after_sync();
          product<4>(tmem + NC * ab, tmem + COL_SLOT + 96u * slot, 32u, dY + (uint64_t)(s * (STAGE >> 4)), YB >> 4, 128u, ID, 4);
          mma_commit_elect(&bars[B_SLFREE + slot]);
          mma_commit_elect(&bars[B_ACC + ab]);
        }
        mma_commit_elect(&bars[B_EMPTY + s]);
      }
    }
    if (*abort_flag != 0) {   // a wait ran out: leave only after the products in flight
      mma_commit_elect(&bars[B_DRAIN]);
      mbar_wait_bounded(&bars[B_DRAIN], 0, WAIT_CYCLES);
    }
  } else if (w >= W_PROD) {
    const int g = (w - W_PROD) >> 2, row = (w & 3) * 32 + lane, f = row & 63;
    const uint32_t addr = tmem + ((uint32_t)((w & 3) * 32) << 16) + COL_SLOT + 16u * g;
    uint32_t seq = 0, k = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x) {
      const Item it = item(idx, P);
      int ca[2], cb[2];   // the two factors' columns
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        int a = 0, b = 0;
        if (it.tile0 + t < LIN) pair_decode(2 * (it.tile0 + t) + (row >> 6), NB, a, b);   // warp-uniform
        ca[t] = it.tile0 + t < LIN ? 8 * a + (f >> 3) : row & 31;
        cb[t] = 8 * b + (f & 7);
      }
      for (int c = 0; c < it.nc; ++c, ++k) {
        const int s = (int)(k % STAGES);
        WAIT(B_FULL + s, k / STAGES, 145);
        const float* x = reinterpret_cast<const float*>(sm + s * STAGE + g * 32 * 128);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (t < it.ntl) {
            uint32_t r[3][16];
            const float *xa = x + ca[t], *xb = x + cb[t];
            if (it.tile0 + t < LIN) {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                split3(mul2(pack2(xa[64 * j], xa[64 * j + 32]), pack2(xb[64 * j], xb[64 * j + 32])), r[0][j], r[1][j], r[2][j]);
            } else if (row < D) {
#pragma unroll
              for (int j = 0; j < 16; ++j) split3(pack2(xa[64 * j], xa[64 * j + 32]), r[0][j], r[1][j], r[2][j]);
            } else {   // the constant feature (rows of Y past the last token are zero), and nothing
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                r[0][j] = row == D ? 0x3F803F80u : 0u;
                r[1][j] = r[2][j] = 0u;
              }
            }
            __syncwarp();
            const uint32_t slot = seq % SLOTS;
            if (seq >= SLOTS) WAIT(B_SLFREE + (int)slot, seq / SLOTS - 1u, 146);
            tc_fence_after_sync();
#pragma unroll
            for (int p = 0; p < 3; ++p) tmem_st16(addr + 96u * slot + 32u * p, r[p]);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[B_SLOT + slot]);
            ++seq;
          }
        }
      }
    }
  } else if (w >= W_DRAIN) {
    const int quarter = w & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    uint32_t seq = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x) {
      const Item it = item(idx, P);
      uint64_t tot[2][17];
#pragma unroll
      for (int j = 0; j < 17; ++j) tot[0][j] = tot[1][j] = 0ull;
      for (int c = 0; c < it.nc; ++c) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (t < it.ntl) {
            const uint32_t ab = seq % ACCS;
            WAIT(B_ACC + (int)ab, seq / ACCS, 147);
            tc_fence_after_sync();
            drain(tot[t], lane_addr + NC * ab, &bars[B_AFREE + ab], lane);
            ++seq;
          }
        }
      }
      // rows -> shared memory -> the state's rows, which lie one behind the other; each warp its own 32
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (t < it.ntl) {
          float4* dst = reinterpret_cast<float4*>(sm + OFF_OUT + (t * 128 + row) * LD * 4);
#pragma unroll
          for (int q = 0; q < 9; ++q) {
            float a, b, c = 0.f, d = 0.f;
            unpack2(tot[t][2 * q], a, b);
            if (q < 8) unpack2(tot[t][q < 8 ? 2 * q + 1 : 0], c, d);
            dst[q] = make_float4(a, b, c, d);
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        for (int t = 0; t < it.ntl; ++t) {
          const int row0 = (it.tile0 + t - P.tile_first) * 128 + quarter * 32, rows = min(32, P.state_rows - row0);
          if (rows > 0)
            bulk_store(P.out + (((long long)it.head * P.nsplit + it.split) * P.state_rows + row0) * LD, sm + OFF_OUT + (t * 128 + quarter * 32) * LD * 4,
                       (uint32_t)(rows * LD * 4));
        }
        bulk_commit_group();
      }
    }
    if (lane == 0) bulk_wait_read_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {   // a wait ran out: copies in flight still land in this block's shared memory
    if (w == W_LOAD)
      for (int i = loaded > STAGES ? loaded - STAGES : 0; i < loaded; ++i) mbar_wait_bounded(&bars[B_FULL + i % STAGES], (uint32_t)(i / STAGES) & 1u, WAIT_CYCLES);
    __syncthreads();
  }
  if (w == W_MMA) tmem_dealloc(tmem, 512);
}
}  // namespace mo

// ---- raw states -> weighted pieces of the state before (reverse: after) each segment ----------------------------------------
// Running sum over the segments, times the polynomial weights, split.  A thread owns (unit, block of eight columns, row) of a
// head; four segments' loads are in flight (one at a time, the sum over 255 segments was a chain of memory latencies).
__global__ void __launch_bounds__(64) pack_kernel(const float* __restrict__ raw, uint8_t* __restrict__ S, float* __restrict__ cst, int ns, int reverse,
                                                  int order, float c0, float c1, float c2) {
  const int u0 = order == 2 ? 0 : NPAIR, u = u0 + blockIdx.x, cb = blockIdx.y, head = blockIdx.z, r = threadIdx.x;
  const int rows = (order == 2 ? 64 * NPAIR : 0) + D + 1;
  const long long step = (long long)rows * LD;
  const float* src = raw + (long long)head * ns * step;
  constexpr int AHEAD = 4;
  if (u == UNITS) {   // the constant row
    if (cb > 0 || r >= CST) return;
    float s = 0.f;
    src += (long long)(rows - 1) * LD + r;
    for (int i0 = 0; i0 < ns; i0 += AHEAD) {
      float v[AHEAD];
#pragma unroll
      for (int e = 0; e < AHEAD; ++e) v[e] = r <= D && i0 + e < ns ? src[(reverse ? ns - 1 - i0 - e : i0 + e) * step] : 0.f;
#pragma unroll
      for (int e = 0; e < AHEAD; ++e) {
        const int i = i0 + e;
        s += v[e];
        if (i < ns) cst[((long long)head * ns + (reverse ? ns - 1 - i : i)) * CST + r] = s * c0;
      }
    }
    return;
  }
  const bool lin = u == NPAIR, live = (!lin || r < D) && cb <= D / 8;
  float wgt = c1;
  if (!lin) {
    int a, b;
    pair_decode(u, NB, a, b);
    wgt = a == b ? c2 : 2.f * c2;
  }
  src += (long long)(64 * (u - u0) + r) * LD + 8 * cb;
  uint8_t* dst = S + ((long long)head * ns * UNITS + u) * UNIT + cb * 1024 + r * 16;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int i0 = 0; i0 < ns; i0 += AHEAD) {
    float4 v[AHEAD][2];
#pragma unroll
    for (int e = 0; e < AHEAD; ++e) {
      v[e][0] = v[e][1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live && i0 + e < ns) {
        const float4* p = reinterpret_cast<const float4*>(src + (reverse ? ns - 1 - i0 - e : i0 + e) * step);
        v[e][0] = p[0];
        if (cb < D / 8) v[e][1] = p[1];
      }
    }
#pragma unroll
    for (int e = 0; e < AHEAD; ++e) {
      const int i = i0 + e;
      s[0] += v[e][0].x; s[1] += v[e][0].y; s[2] += v[e][0].z; s[3] += v[e][0].w;
      s[4] += v[e][1].x; s[5] += v[e][1].y; s[6] += v[e][1].z; s[7] += v[e][1].w;
      const int k = reverse ? ns - 1 - i : i;
      if (i < ns) {
        uint32_t o[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split3(pack2(s[2 * j] * wgt, s[2 * j + 1] * wgt), o[0][j], o[1][j], o[2][j]);
        if (cb == D / 8) {   // piece 0: the column that counts, and the pieces as the chain kernel pairs them with G's
          const uint32_t hi = o[0][0] & 0xffffu, mid = o[1][0] & 0xffffu, lo = o[2][0] & 0xffffu;
          o[0][0] = hi | hi << 16;
          o[0][1] = mid | hi << 16;
          o[0][2] = mid | lo << 16;
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
          *reinterpret_cast<uint4*>(dst + (long long)k * UNITS * UNIT + p * PIECE) = make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]);
      }
    }
  }
}

// ---- apply: out = (partial + Phi(x) S) [/ denominator], the partial result being in `out` already ---------------------------
namespace ap {
constexpr int THREADS = 512, W_MMA = 0, W_LOAD = 1, W_DRAIN = 4, W_PROD = 8;
constexpr int S_STAGES = 4;
constexpr int OFF_X = 0, OFF_P = 4 * LT, OFF_S = OFF_P + 2 * LT, OFF_BAR = OFF_S + S_STAGES * UNIT, BYTES = OFF_BAR + 512 + 1024;
static_assert(BYTES <= 232448 && UNIT % 1024 == 0, "shared memory budget");
constexpr int B_XFULL = 0, B_XFREE = 2, B_SFULL = 4, B_SEMPTY = B_SFULL + S_STAGES, B_SLOT = B_SEMPTY + S_STAGES, B_SLFREE = B_SLOT + SLOTS,
              B_ACC = B_SLFREE + SLOTS, B_AFREE = B_ACC + ACCS, B_PFULL = B_AFREE + ACCS, B_PFREE = B_PFULL + 1, B_DRAIN = B_PFREE + 1, B_COUNT = B_DRAIN + 1;

template <bool FWD>
__global__ void __launch_bounds__(THREADS, 1) apply_kernel(const __grid_constant__ lng::Maps M, const lng::Params P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      uint32_t n = 1;
      if (i >= B_XFREE && i < B_XFREE + 2) n = 8;
      if ((i >= B_SLOT && i < B_SLFREE) || (i >= B_AFREE && i < B_PFULL) || i == B_PFREE) n = 4;
      mbar_init(&bars[i], n);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (w == W_MMA) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto WAIT = [&](int bar, uint32_t phase, int code) { wait_fast(&bars[bar], phase & 1u, code, abort_flag); };
  const int u0 = P.u0, units = UNITS - u0;

  int xs = 0, parts = 0, ss = 0;   // what the loader has asked for
  if (w == W_LOAD) {
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      if (n >= 2) WAIT(B_XFREE + (n & 1), (uint32_t)(n >> 1) - 1u, 150);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        uint64_t* bar = &bars[B_XFULL + (n & 1)];
        mbar_arrive_expect_tx(bar, 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + ((n & 1) * 2 + m) * LT, &M.x, bar, 0, k.tok + m * 128, k.h, k.b);
      }
      xs = n + 1;
      const uint8_t* src = P.S + ((long long)k.st * UNITS + u0) * UNIT;
      for (int j = 0; j < units; ++j, ++ss) {
        const int s = ss % S_STAGES;
        if (ss >= S_STAGES) WAIT(B_SEMPTY + s, (uint32_t)(ss / S_STAGES) - 1u, 151);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&bars[B_SFULL + s], UNIT);
          bulk_load(sm + OFF_S + s * UNIT, src + (long long)j * UNIT, UNIT, &bars[B_SFULL + s]);
        }
      }
      if (n >= 1) WAIT(B_PFREE, (uint32_t)n - 1u, 152);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_PFULL], 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + OFF_P + m * LT, &M.part, &bars[B_PFULL], 0, k.tok + m * 128, k.h, k.b);
      }
      parts = n + 1;
    }
  } else if (w == W_MMA) {
    constexpr uint32_t ID = make_idesc_bf16(128, NC, 0, 1);
    uint32_t seq = 0, sg = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x) {
      for (int j = 0; j < units; ++j, ++sg) {
        const uint32_t s = sg % S_STAGES;
        WAIT(B_SFULL + (int)s, sg / S_STAGES, 154);
        const uint64_t dS = make_smem_desc(smem_u32(sm + OFF_S) + s * UNIT, 128, 1024, 0);
        const int kk_used = j == units - 1 ? 2 : 4;   // the linear unit: 32 features
        for (int m = 0; m < 2; ++m, ++seq) {
          const uint32_t slot = seq % SLOTS, ab = seq % ACCS;
          WAIT(B_SLOT + (int)slot, seq / SLOTS, 155);
          if (seq >= ACCS) WAIT(B_AFREE + (int)ab, seq / ACCS - 1u, 153);
          tc_fence_after_sync();
          product<4>(tmem + NC * ab, tmem + COL_SLOT + 96u * slot, 32u, dS, PIECE >> 4, 16u, ID, kk_used);
          mma_commit_elect(&bars[B_SLFREE + slot]);
          mma_commit_elect(&bars[B_ACC + ab]);
        }
        mma_commit_elect(&bars[B_SEMPTY + s]);
      }
    }
    if (*abort_flag != 0) {
      mma_commit_elect(&bars[B_DRAIN]);
      mbar_wait_bounded(&bars[B_DRAIN], 0, WAIT_CYCLES);
    }
  } else if (w >= W_PROD) {   // one warpgroup per tile; thread = token
    const int m = (w - W_PROD) >> 2, row = (w & 3) * 32 + lane, sw = row & 7;
    const uint32_t addr = tmem + ((uint32_t)((w & 3) * 32) << 16) + COL_SLOT;
    uint32_t seq = (uint32_t)m;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      WAIT(B_XFULL + (n & 1), (uint32_t)(n >> 1), 156);
      const uint8_t* x = sm + ((n & 1) * 2 + m) * LT + row * 128;
      auto block = [&](int c, uint64_t (&v)[4]) {   // the eight values of block c, in pairs
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(x + (((2 * c) ^ sw) << 4)), q = *reinterpret_cast<const ulonglong2*>(x + (((2 * c + 1) ^ sw) << 4));
        v[0] = p.x; v[1] = p.y; v[2] = q.x; v[3] = q.y;
      };
      int a = u0 > 0 ? NB : 0, b = 0;
      for (int j = 0; j < units; ++j, seq += 2u) {
        const uint32_t slot = seq % SLOTS, base = addr + 96u * slot;
        if (seq >= SLOTS) WAIT(B_SLFREE + (int)slot, seq / SLOTS - 1u, 157);
        tc_fence_after_sync();
        if (a < NB) {
          uint64_t xa[4], xb[4];
          block(a, xa);
          block(b, xb);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[3][16];
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
              float lo, hi;
              unpack2(xa[2 * h + (i4 >> 1)], lo, hi);
              const float v = (i4 & 1) ? hi : lo;
              const uint64_t vv = pack2(v, v);
#pragma unroll
              for (int c = 0; c < 4; ++c) split3(mul2(vv, xb[c]), r[0][4 * i4 + c], r[1][4 * i4 + c], r[2][4 * i4 + c]);
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) tmem_st16(base + 32u * p + 16u * h, r[p]);
          }
          if (++b == NB) { ++a; b = a; }
        } else {   // the linear unit
          uint32_t r[3][16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint64_t v[4];
            block(c, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) split3(v[e], r[0][4 * c + e], r[1][4 * c + e], r[2][4 * c + e]);
          }
#pragma unroll
          for (int p = 0; p < 3; ++p) tmem_st16(base + 32u * p, r[p]);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[B_SLOT + slot]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_XFREE + (n & 1)]);
    }
  } else if (w >= W_DRAIN) {
    const int quarter = w & 3, sw = lane & 7;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    uint32_t seq = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      uint64_t tot[2][17];
      {   // the constant row
        const ulonglong2* cst = reinterpret_cast<const ulonglong2*>(P.cst + (long long)k.st * CST);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const ulonglong2 c = __ldg(cst + q);
          tot[0][2 * q] = tot[1][2 * q] = c.x;
          tot[0][2 * q + 1] = tot[1][2 * q + 1] = c.y;
        }
        tot[0][16] = tot[1][16] = __ldg(cst + 8).x;
      }
      for (int j = 0; j < units; ++j) {
#pragma unroll
        for (int m = 0; m < 2; ++m, ++seq) {
          const uint32_t ab = seq % ACCS;
          WAIT(B_ACC + (int)ab, seq / ACCS, 158);
          tc_fence_after_sync();
          drain(tot[m], lane_addr + NC * ab, &bars[B_AFREE + ab], lane);
        }
      }
      WAIT(B_PFULL, (uint32_t)n, 159);
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int row = k.tok + m * 128 + quarter * 32 + lane;
        uint8_t* own = sm + OFF_P + m * LT + (quarter * 32 + lane) * 128;
        float wgt = 1.f;
        if (FWD) {
          float gs, unused;
          unpack2(tot[m][16], gs, unused);
          if (row < P.n) {
            float* g = reinterpret_cast<float*>(const_cast<void*>(P.g.ptr)) + (long long)k.b * P.g.sb + (long long)k.h * P.g.sh + (long long)row * P.g.sn;
            gs += *g;
            *g = gs;
          }
          wgt = 1.f / gs;
        }
        const uint64_t ww = pack2(wgt, wgt);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          ulonglong2* at = reinterpret_cast<ulonglong2*>(own + ((q ^ sw) << 4));
          const ulonglong2 p = *at;
          ulonglong2 o;
          o.x = add2(tot[m][2 * q], p.x);
          o.y = add2(tot[m][2 * q + 1], p.y);
          if (FWD) {
            o.x = mul2(o.x, ww);
            o.y = mul2(o.y, ww);
          }
          *at = o;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row < P.n) {
          tma_store_4d(&M.out, own, 0, row, k.h, k.b);
          bulk_commit_group();
        }
      }
      if (lane == 0) {
        bulk_wait_read_all();
        mbar_arrive(&bars[B_PFREE]);
      }
      __syncwarp();
    }
    if (lane == 0) bulk_wait_read_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    if (w == W_LOAD) {
      for (int i = xs > 2 ? xs - 2 : 0; i < xs; ++i) mbar_wait_bounded(&bars[B_XFULL + (i & 1)], (uint32_t)(i >> 1) & 1u, WAIT_CYCLES);
      for (int i = ss > S_STAGES ? ss - S_STAGES : 0; i < ss; ++i) mbar_wait_bounded(&bars[B_SFULL + i % S_STAGES], (uint32_t)(i / S_STAGES) & 1u, WAIT_CYCLES);
      if (parts > 0) mbar_wait_bounded(&bars[B_PFULL], (uint32_t)(parts - 1) & 1u, WAIT_CYCLES);
    }
    __syncthreads();
  }
  if (w == W_MMA) tmem_dealloc(tmem, 512);
}
}  // namespace ap

// ---- chain: out += sum_u chain rule through Phi of dphi_u, dphi_u = G S_u^T (see long_kernels.cuh) ---------------------------
// The six piece products of the denominator column share one K = 16 step: [hi mid hi lo mid hi] of G against [hi hi mid hi mid lo]
// of S: 13 MMAs per unit instead of 18, and G of two items fits into TMEM, so the next item's is there before this one's
// products end.
namespace ch {
constexpr int THREADS = 384, W_LOAD = 2, W_CHAIN = 4;
constexpr int S_STAGES = 3;
constexpr int GT = 128 * NC * 2;              // one piece of a G tile: rows of 48 columns, not swizzled
constexpr int OFF_X = 0, OFF_P = 4 * LT, OFF_G = OFF_P + 2 * LT, OFF_S = OFF_G + 6 * GT, OFF_BAR = OFF_S + S_STAGES * UNIT, BYTES = OFF_BAR + 512 + 1024;
static_assert(BYTES <= 232448, "shared memory budget");
constexpr int B_XFULL = 0, B_XFREE = 2, B_GFULL = 4, B_GFREE = 5, B_GT = 6, B_SFULL = 8, B_SEMPTY = B_SFULL + S_STAGES,
              B_D = B_SEMPTY + S_STAGES, B_DFREE = B_D + 4, B_PFULL = B_DFREE + 4, B_PFREE = B_PFULL + 1, B_DRAIN = B_PFREE + 1, B_COUNT = B_DRAIN + 2;
constexpr uint32_t COL_D = 224;   // dphi: tile m, buffer b at COL_D + 128 m + 64 b
constexpr uint32_t G_TILE = 56;    // G of item n, tile m at 112 (n & 1) + 56 m: three pieces of 16 columns, the tail of 8

__global__ void __launch_bounds__(THREADS, 1) chain_kernel(const __grid_constant__ lng::Maps M, const lng::Params P) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      uint32_t n = 1;
      if (i == B_XFREE || i == B_XFREE + 1 || i == B_GFREE || i == B_PFREE) n = 8;
      if (i == B_GT || i == B_GT + 1 || (i >= B_DFREE && i < B_DFREE + 4)) n = 4;
      if (i >= B_SEMPTY && i < B_SEMPTY + S_STAGES) n = 2;
      mbar_init(&bars[i], n);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (w == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto WAIT = [&](int bar, uint32_t phase, int code) { wait_fast(&bars[bar], phase & 1u, code, abort_flag); };
  const int u0 = P.u0, units = UNITS - u0;

  int xs = 0, gs = 0, parts = 0, ss = 0;
  if (w == W_LOAD) {
    // x and G of item n (of this block), as soon as the last users have let go
    auto load_item = [&](int idx, int n) {
      const Work k = work(idx, P);
      if (n >= 2) WAIT(B_XFREE + (n & 1), (uint32_t)(n >> 1) - 1u, 160);
      if (n >= 1) WAIT(B_GFREE, (uint32_t)n - 1u, 161);
      if (*abort_flag != 0) return;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_GFULL], 6 * GT);
        for (int i = 0; i < 6; ++i) tma_load_4d(sm + OFF_G + i * GT, &M.y, &bars[B_GFULL], 0, k.tok + (i / 3) * 128, k.head, i % 3);
        uint64_t* bar = &bars[B_XFULL + (n & 1)];
        mbar_arrive_expect_tx(bar, 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + ((n & 1) * 2 + m) * LT, &M.x, bar, 0, k.tok + m * 128, k.h, k.b);
      }
      xs = gs = n + 1;
    };
    int n = 0;
    if ((int)blockIdx.x < P.nitems) load_item(blockIdx.x, 0);
    const int ahead = min(3, units - 1);   // unit after which the next item's tiles are asked for: the chain warps take G later
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      const uint8_t* src = P.S + ((long long)k.st * UNITS + u0) * UNIT;
      for (int j = 0; j < units; ++j, ++ss) {
        const int s = ss % S_STAGES;
        if (ss >= S_STAGES) WAIT(B_SEMPTY + s, (uint32_t)(ss / S_STAGES) - 1u, 162);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&bars[B_SFULL + s], UNIT);
          bulk_load(sm + OFF_S + s * UNIT, src + (long long)j * UNIT, UNIT, &bars[B_SFULL + s]);
        }
        if (j == ahead && idx + (int)gridDim.x < P.nitems) load_item(idx + gridDim.x, n + 1);
      }
      if (n >= 1) WAIT(B_PFREE, (uint32_t)n - 1u, 163);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_PFULL], 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + OFF_P + m * LT, &M.part, &bars[B_PFULL], 0, k.tok + m * 128, k.h, k.b);
      }
      parts = n + 1;
    }
  } else if (w < 2) {
    constexpr uint32_t ID = make_idesc_bf16(128, 64, 0, 0);
    uint32_t sg = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      WAIT(B_GT + w, (uint32_t)n, 164);
      for (int j = 0; j < units; ++j, ++sg) {
        const uint32_t s = sg % S_STAGES, buf = sg & 1u;
        WAIT(B_SFULL + (int)s, sg / S_STAGES, 165);
        if (sg >= 2) WAIT(B_DFREE + 2 * w + (int)buf, (sg >> 1) - 1u, 166);
        tc_fence_after_sync();
        const uint64_t dS = make_smem_desc(smem_u32(sm + OFF_S) + s * UNIT, 1024, 128, 0);
        const uint32_t acc = tmem + COL_D + 128u * w + 64u * buf, ga = tmem + G_TILE * (2u * (n & 1) + w);
        product<2>(acc, ga, 16u, dS, PIECE >> 4, 128u, ID, 2);
        mma_ts_elect(acc, ga + 48u, dS + (uint64_t)256, ID, 1u);
        mma_commit_elect(&bars[B_D + 2 * w + buf]);
        mma_commit_elect(&bars[B_SEMPTY + s]);
      }
    }
    if (*abort_flag != 0) {
      mma_commit_elect(&bars[B_DRAIN + w]);
      mbar_wait_bounded(&bars[B_DRAIN + w], 0, WAIT_CYCLES);
    }
  } else if (w >= W_CHAIN) {
    const int m = (w - W_CHAIN) >> 2, quarter = w & 3, l = quarter * 32 + lane, sw = lane & 7;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    auto take_g = [&](int n) {   // G of item n: shared memory -> TMEM
      WAIT(B_GFULL, (uint32_t)n, 167);
      const uint32_t dst = lane_addr + G_TILE * (2u * (n & 1) + m);
      uint32_t tail[3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const uint4* src = reinterpret_cast<const uint4*>(sm + OFF_G + (3 * m + p) * GT + l * (NC * 2));
        uint32_t r[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 v = src[c];
          r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
        }
        tail[p] = src[4].x & 0xffffu;
        tmem_st16(dst + 16u * p, r);
      }
      const uint32_t r8[8] = {tail[0] | tail[1] << 16, tail[0] | tail[2] << 16, tail[1] | tail[0] << 16, 0u, 0u, 0u, 0u, 0u};
      tmem_st8(dst + 48u, r8);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bars[B_GT + m]);
        mbar_arrive(&bars[B_GFREE]);
      }
    };
    if ((int)blockIdx.x < P.nitems) take_g(0);
    uint32_t sg = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      const int row = k.tok + m * 128 + l;
      WAIT(B_XFULL + (n & 1), (uint32_t)(n >> 1), 168);
      const uint8_t* x = sm + ((n & 1) * 2 + m) * LT + l * 128;
      uint64_t acc[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[i] = 0ull;
      auto block = [&](int c, uint64_t (&v)[4]) {   // the eight values of block c of this token's row, in pairs
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(x + (((2 * c) ^ sw) << 4)), q = *reinterpret_cast<const ulonglong2*>(x + (((2 * c + 1) ^ sw) << 4));
        v[0] = p.x; v[1] = p.y; v[2] = q.x; v[3] = q.y;
      };
      auto next_unit = [&]() -> uint32_t {   // waits for the unit's dphi; its TMEM address
        const uint32_t buf = sg & 1u;
        WAIT(B_D + 2 * m + (int)buf, sg >> 1, 169);
        tc_fence_after_sync();
        return lane_addr + COL_D + 128u * m + 64u * buf;
      };
      auto unit_done = [&] {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[B_DFREE + 2 * m + (int)(sg & 1u)]);
        ++sg;
      };
      if (u0 == 0) {
#pragma unroll
        for (int a = 0; a < NB; ++a) {
          if (a == 1 && idx + (int)gridDim.x < P.nitems) take_g(n + 1);
          uint64_t xa[4], t[8];
          block(a, xa);
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = 0ull;
#pragma unroll
          for (int b = a; b < NB; ++b) {
            uint64_t xb[4];
            block(b, xb);
            const uint32_t addr = next_unit();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t d[32];
              tmem_ld32(addr + 32u * h, d);
              tmem_ld_wait();
              if (h == 1) unit_done();
#pragma unroll
              for (int i4 = 0; i4 < 4; ++i4) {
                const int i = 4 * h + i4;
                float lo, hi;
                unpack2(xa[i >> 1], lo, hi);
                const float xi = (i & 1) ? hi : lo;
                const uint64_t xx = pack2(xi, xi);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const uint64_t dp = pack2u(d[8 * i4 + 2 * j], d[8 * i4 + 2 * j + 1]);
                  t[i] = fma2(dp, xb[j], t[i]);
                  acc[4 * b + j] = fma2(dp, xx, acc[4 * b + j]);
                }
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float a0, a1, b0, b1;
            unpack2(t[2 * i], a0, a1);
            unpack2(t[2 * i + 1], b0, b1);
            acc[4 * a + i] = add2(acc[4 * a + i], pack2(a0 + a1, b0 + b1));
          }
        }
      }
      if (u0 > 0 && idx + (int)gridDim.x < P.nitems) take_g(n + 1);
      {   // the linear unit
        const uint32_t addr = next_unit();
        uint32_t d[32];
        tmem_ld32(addr, d);
        tmem_ld_wait();
        unit_done();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j] = add2(acc[j], pack2u(d[2 * j], d[2 * j + 1]));
      }
      if (lane == 0) mbar_arrive(&bars[B_XFREE + (n & 1)]);
      uint8_t* own = sm + OFF_P + m * LT + l * 128;
      WAIT(B_PFULL, (uint32_t)n, 170);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        ulonglong2* at = reinterpret_cast<ulonglong2*>(own + ((q ^ sw) << 4));
        const ulonglong2 p = *at;
        ulonglong2 o;
        o.x = add2(acc[2 * q], p.x);
        o.y = add2(acc[2 * q + 1], p.y);
        *at = o;
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && row < P.n) {
        tma_store_4d(&M.out, own, 0, row, k.h, k.b);
        bulk_commit_group();
      }
      if (lane == 0) {
        bulk_wait_read_all();
        mbar_arrive(&bars[B_PFREE]);
      }
      __syncwarp();
    }
    if (lane == 0) bulk_wait_read_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    if (w == W_LOAD) {
      for (int i = xs > 2 ? xs - 2 : 0; i < xs; ++i) mbar_wait_bounded(&bars[B_XFULL + (i & 1)], (uint32_t)(i >> 1) & 1u, WAIT_CYCLES);
      if (gs > 0) mbar_wait_bounded(&bars[B_GFULL], (uint32_t)(gs - 1) & 1u, WAIT_CYCLES);
      for (int i = ss > S_STAGES ? ss - S_STAGES : 0; i < ss; ++i) mbar_wait_bounded(&bars[B_SFULL + i % S_STAGES], (uint32_t)(i / S_STAGES) & 1u, WAIT_CYCLES);
      if (parts > 0) mbar_wait_bounded(&bars[B_PFULL], (uint32_t)(parts - 1) & 1u, WAIT_CYCLES);
    }
    __syncthreads();
  }
  if (w == 0) tmem_dealloc(tmem, 512);
}
}  // namespace ch

}  // namespace f32
