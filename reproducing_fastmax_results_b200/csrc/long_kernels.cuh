// Long sequences, bf16: the tokens a query sees are cut at a window boundary.  Keys of its own window are evaluated pair by
// pair (pair_kernel with Params::window); everything before the window enters through the moment state S of those keys,
//     O' += Phi(q) S,      dq += Phi'(q) (S dO'),      dv += Phi(k) dS,      dk += Phi'(k) (dS [v | 1])
// (dS: gradient moments of the queries after the key's window).  A state is constant within a window, so nothing here is a
// scan: every 256-token item is independent, one thread block per SM walks over them, and each result is finished here and
// written once.  Without a mask there are no pairs and one state per head.  Included by pair_kernels.cu inside fm.
//
// Measured, 8 heads of 131072 x 64, forward + backward: 7.9 ms by segmented scans (their serial chains and float32 partial sums in
// memory), 4.0 to 4.5 here from box to box; of 4.1: moments 2 x 495 us, pairs 230 + 740, apply 2 x 295, chain rule 380 + 370,
// packing 2 x 156.
#pragma once

namespace lng {

using namespace tc;
using pair::bf16x2;
using pair::Item;
using pair::fma2;
using pair::add2;
using pair::mul2;
using pair::pack2;
using pair::pack2u;
using pair::unpack2;
using pair::tmem_ld;
using pair::wait_fast;
using pair::WAIT_CYCLES;

constexpr int ROWS = 256;               // tokens of an item: two tiles of 128
constexpr int LT = 128 * 128;           // a tile of 128 rows of 128 bytes

template <int D>
struct Geo {
  static constexpr int NB = D / 8;
  static constexpr int NPAIR = NB * (NB + 1) / 2;
  static constexpr int UNITS = NPAIR + 1;              // pair units and the linear unit; the constant row is added by the epilogue
  static constexpr int CB = D / 8 + 2;                 // 8-column blocks: values, [denominator, 0 ...], 0
  static constexpr int UNIT_BYTES = CB * 1024;         // [block][64 rows][8 columns] bf16
  static constexpr int CST = D + 8;                    // constant row, float32
  static constexpr int STATE_LD = D + 4;
};

struct Params {
  const uint8_t* S;          // packed states [head][ns][UNITS][UNIT_BYTES]
  const float* cst;          // [head][ns][CST]
  const float* ndelta;       // chain, dq: -delta per query, [head][nd_ld]
  View g;                    // apply forward: denominators, partial in, final out
  int nd_ld;
  int heads, n;              // tokens
  int row0, seg, ns;         // token r (>= row0) uses state (r - row0) / seg
  int items_per_head, nitems;
  int u0;                    // first unit (order 1: the linear unit alone)
  int part;                  // there is a partial result to add
  float w1;                  // factor of the partial denominators
};
struct Maps {
  CUtensorMap x;             // q or k
  CUtensorMap y;             // chain: dO' or v
  CUtensorMap part;          // float32 partial result, 32-column boxes
  CUtensorMap out;           // 32-row boxes
};

struct Work {
  int head, b, h, tok, st;   // st: state index
};
__device__ __forceinline__ Work work(int idx, const Params& P) {
  Work w;
  w.head = idx / P.items_per_head;
  w.tok = P.row0 + (idx - w.head * P.items_per_head) * ROWS;
  w.b = w.head / P.heads;
  w.h = w.head - w.b * P.heads;
  w.st = w.head * P.ns + (w.tok - P.row0) / P.seg;
  return w;
}

// ---- apply: out = (partial + Phi(x) S) [/ denominator] --------------------------------------------------------------------
// Warp roles: 0 MMA issuer, 1 loader, 4-7 epilogue, 8-15 producers (one warpgroup per tile).  A slab of 128 features goes
// through a ring of three 64-column TMEM slots shared by the two tiles; accumulators are double-buffered, so the epilogue of an
// item runs under the products of the next.  Bound by the tensor pipe (A from TMEM, N = D + 16: 43 clocks per 16 features and
// tile at D = 64).
namespace ap {
constexpr int THREADS = 512, W_MMA = 0, W_LOAD = 1, W_EPI = 4, W_PROD = 8;
constexpr int S_STAGES = 4;
template <int D>
struct Lay {
  static constexpr int SLABS = (Geo<D>::UNITS + 1) / 2;
  static constexpr int S_STAGE = 2 * Geo<D>::UNIT_BYTES;
  static constexpr int OFF_X = 0;                              // two items x two tiles
  static constexpr int OFF_P = 4 * LT;                   // partial result of two tiles, later the output rows
  static constexpr int OFF_S = OFF_P + 2 * (D / 32) * LT;
  static constexpr int OFF_BAR = OFF_S + S_STAGES * S_STAGE;
  static constexpr int BYTES = OFF_BAR + 512 + 1024;
  static_assert(BYTES <= 232448, "shared memory budget");
};
constexpr int B_XFULL = 0, B_XFREE = 2, B_SFULL = 4, B_SEMPTY = B_SFULL + S_STAGES, B_SLOT = B_SEMPTY + S_STAGES, B_SLFREE = B_SLOT + 3,
              B_ACC = B_SLFREE + 3, B_AFREE = B_ACC + 2, B_PFULL = B_AFREE + 2, B_PFREE = B_PFULL + 1, B_DRAIN = B_PFREE + 1, B_COUNT = B_DRAIN + 1;
constexpr uint32_t COL_SLOT = 320;

template <int D, bool FWD>
__global__ void __launch_bounds__(THREADS, 1) apply_kernel(const __grid_constant__ Maps M, const Params P) {
  using L = Lay<D>;
  using G = Geo<D>;
  constexpr int NC = D + 16;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + L::OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L::OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L::OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      uint32_t n = 1;
      if (i >= B_XFREE && i < B_XFREE + 2) n = 8;
      if ((i >= B_SLOT && i < B_SLFREE) || (i >= B_AFREE && i < B_AFREE + 2) || i == B_PFREE) n = 4;
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
  const int u0 = P.u0, slabs = (G::UNITS - u0 + 1) / 2;
  auto units_of = [&](int j) { return min(2, G::UNITS - u0 - 2 * j); };

  int xs = 0, parts = 0, ss = 0;   // what the loader has asked for
  if (w == W_LOAD) {
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      if (n >= 2) WAIT(B_XFREE + (n & 1), (uint32_t)(n >> 1) - 1u, 120);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        uint64_t* bar = &bars[B_XFULL + (n & 1)];
        mbar_arrive_expect_tx(bar, 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + ((n & 1) * 2 + m) * LT, &M.x, bar, 0, k.tok + m * 128, k.h, k.b);
      }
      xs = n + 1;
      const uint8_t* src = P.S + ((long long)k.st * G::UNITS + u0) * G::UNIT_BYTES;
      for (int j = 0; j < slabs; ++j, ++ss) {
        const int s = ss % S_STAGES;
        if (ss >= S_STAGES) WAIT(B_SEMPTY + s, (uint32_t)(ss / S_STAGES) - 1u, 121);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          const uint32_t bytes = (uint32_t)(units_of(j) * G::UNIT_BYTES);
          mbar_arrive_expect_tx(&bars[B_SFULL + s], bytes);
          bulk_load(sm + L::OFF_S + s * L::S_STAGE, src + (long long)j * L::S_STAGE, bytes, &bars[B_SFULL + s]);
        }
      }
      if (P.part) {
        if (n >= 1) WAIT(B_PFREE, (uint32_t)n - 1u, 122);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&bars[B_PFULL], 2 * (D / 32) * LT);
          for (int m = 0; m < 2; ++m)
            for (int c = 0; c < D / 32; ++c)
              tma_load_4d(sm + L::OFF_P + (m * (D / 32) + c) * LT, &M.part, &bars[B_PFULL], 32 * c, k.tok + m * 128, k.head, 0);
        }
        parts = n + 1;
      }
    }
  } else if (w == W_MMA) {
    constexpr uint32_t ID = make_idesc_bf16(128, NC, 0, 1);
    uint32_t seq = 0, sg = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const uint32_t buf = (uint32_t)n & 1u;
      if (n >= 2) WAIT(B_AFREE + (int)buf, (uint32_t)(n >> 1) - 1u, 123);
      for (int j = 0; j < slabs; ++j, ++sg) {
        const uint32_t s = sg % S_STAGES;
        WAIT(B_SFULL + (int)s, sg / S_STAGES, 124);
        const int nu = units_of(j);
        const uint64_t dS = make_smem_desc(smem_u32(sm + L::OFF_S) + s * L::S_STAGE, 128, 1024, 0);
#pragma unroll
        for (int m = 0; m < 2; ++m, ++seq) {
          const uint32_t slot = seq % 3u;
          WAIT(B_SLOT + (int)slot, seq / 3u, 125);
          tc_fence_after_sync();
          const uint32_t a = tmem + COL_SLOT + 64u * slot, acc = tmem + (uint32_t)NC * (2u * buf + m);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) mma_ts_elect(acc, a + 8u * kk, dS + (uint64_t)(16 * kk), ID, (j > 0 || kk > 0) ? 1u : 0u);
          if (nu == 2) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) mma_ts_elect(acc, a + 32u + 8u * kk, dS + (uint64_t)((G::UNIT_BYTES >> 4) + 16 * kk), ID, 1u);
          }
          mma_commit_elect(&bars[B_SLFREE + slot]);
        }
        mma_commit_elect(&bars[B_SEMPTY + s]);
      }
      mma_commit_elect(&bars[B_ACC + buf]);
    }
    if (*abort_flag != 0) {   // a wait ran out: leave only after the products in flight
      mma_commit_elect(&bars[B_DRAIN]);
      mbar_wait_bounded(&bars[B_DRAIN], 0, WAIT_CYCLES);
    }
  } else if (w >= W_PROD) {
    const int m = (w - W_PROD) >> 2, row = (w & 3) * 32 + lane;
    const uint32_t addr = tmem + ((uint32_t)((w & 3) * 32) << 16) + COL_SLOT;
    uint32_t seq = (uint32_t)m;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      WAIT(B_XFULL + (n & 1), (uint32_t)(n >> 1), 126);
      const uint8_t* x = sm + ((n & 1) * 2 + m) * LT;
      int a = 0, b = 0;
      if (u0 > 0) a = G::NB;
      for (int j = 0; j < slabs; ++j, seq += 2u) {
        const uint32_t slot = seq % 3u;
        if (seq >= 3u) WAIT(B_SLFREE + (int)slot, seq / 3u - 1u, 127);
        tc_fence_after_sync();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          if (a < G::NB) {
            apply_pair_slab(r, x, row, a, b, false);
            if (++b == G::NB) { ++a; b = a; }
            tmem_st32(addr + 64u * slot + 32u * h, r);
          } else if (a == G::NB) {   // the linear unit
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint4 v = c < D / 8 ? sw_chunk(x, row, c) : make_uint4(0u, 0u, 0u, 0u);
              r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
            }
            ++a;
            tmem_st32(addr + 64u * slot + 32u * h, r);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[B_SLOT + slot]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_XFREE + (n & 1)]);
    }
  } else if (w >= W_EPI) {
    const int quarter = w & 3;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      const float4* cst = reinterpret_cast<const float4*>(P.cst + (long long)k.st * G::CST);
      float* g = reinterpret_cast<float*>(const_cast<void*>(P.g.ptr)) + (FWD ? (long long)k.b * P.g.sb + (long long)k.h * P.g.sh : 0);
      WAIT(B_ACC + (n & 1), (uint32_t)(n >> 1), 128);
      if (P.part) WAIT(B_PFULL, (uint32_t)n, 129);
      tc_fence_after_sync();
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int row = k.tok + m * 128 + quarter * 32 + lane;
        const uint32_t acc = lane_addr + (uint32_t)NC * (2u * (n & 1) + m);
        uint8_t* own = sm + L::OFF_P + m * (D / 32) * LT + (quarter * 32 + lane) * 128;
        const int sw = lane & 7;
        float wgt = 1.f;
        if (FWD) {
          uint32_t r8[8];
          tmem_ld8(acc + (uint32_t)D, r8);
          tmem_ld_wait();
          float gs = __uint_as_float(r8[0]) + __ldg(P.cst + (long long)k.st * G::CST + D);
          if (row < P.n) {
            if (P.part) gs += g[(long long)row * P.g.sn];   // (final factor already in)
            g[(long long)row * P.g.sn] = gs;
          }
          wgt = 1.f / gs;
        }
        uint32_t o[D / 2];
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(acc + 32u * c, r);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const float4 cc = __ldg(cst + 8 * c + q);
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            if (P.part) p = *reinterpret_cast<const float4*>(own + c * LT + ((q ^ sw) << 4));
            o[16 * c + 2 * q] = bf16x2((__uint_as_float(r[4 * q]) + cc.x + p.x) * wgt, (__uint_as_float(r[4 * q + 1]) + cc.y + p.y) * wgt);
            o[16 * c + 2 * q + 1] = bf16x2((__uint_as_float(r[4 * q + 2]) + cc.z + p.z) * wgt, (__uint_as_float(r[4 * q + 3]) + cc.w + p.w) * wgt);
          }
        }
        if (m == 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[B_AFREE + (n & 1)]);
        }
        if (!P.part && n > 0 && m == 0) {   // the rows staged for the last item have been read (with a partial: see below)
          if (lane == 0) bulk_wait_read_all();
          __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < D / 8; ++q)
          *reinterpret_cast<uint4*>(own + ((q ^ sw) << 4)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row < P.n) {
          tma_store_4d(&M.out, own, 0, row, k.h, k.b);
          bulk_commit_group();
        }
      }
      if (P.part) {
        if (lane == 0) {
          bulk_wait_read_all();
          mbar_arrive(&bars[B_PFREE]);
        }
        __syncwarp();
      }
    }
    if (lane == 0) bulk_wait_read_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {   // a wait ran out: copies in flight still land in this block's shared memory
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

// ---- chain: out = partial + sum_u chain rule through Phi of dphi_u, dphi_u = G S_u^T ---------------------------------------
// G: [dO' | -delta] (dq) or [v | 1] (dk), put into tensor memory once per item; dphi of a 64-feature unit lands in one of two
// TMEM buffers per tile and is contracted with the token's row on CUDA cores: 64 packed multiply-adds per unit and thread,
// accumulators in registers (units are unrolled so that their blocks are static).
// Warp roles: 0, 1 MMA issuers (one per tile), 2 loader, 4-11 chain rule (thread = token).
namespace ch {
constexpr int THREADS = 384, W_LOAD = 2, W_CHAIN = 4;
constexpr int S_STAGES = 5;
template <int D>
struct Lay {
  static constexpr int OFF_X = 0;                              // two items x two tiles
  static constexpr int OFF_G = 4 * LT;                         // one item x two tiles
  static constexpr int OFF_P = OFF_G + 2 * LT;
  static constexpr int OFF_S = OFF_P + 2 * (D / 32) * LT;
  static constexpr int OFF_BAR = OFF_S + S_STAGES * Geo<D>::UNIT_BYTES;
  static constexpr int BYTES = OFF_BAR + 512 + 1024;
  static_assert(BYTES <= 232448, "shared memory budget");
};
constexpr int B_XFULL = 0, B_XFREE = 2, B_GFULL = 4, B_GFREE = 5, B_GT = 6, B_SFULL = 8, B_SEMPTY = B_SFULL + S_STAGES,
              B_D = B_SEMPTY + S_STAGES, B_DFREE = B_D + 4, B_PFULL = B_DFREE + 4, B_PFREE = B_PFULL + 1, B_DRAIN = B_PFREE + 1, B_COUNT = B_DRAIN + 2;
constexpr uint32_t COL_D = 256;   // dphi: tile m, buffer b at COL_D + 128 m + 64 b; G of tile m at 64 m

template <int D, bool DK>
__global__ void __launch_bounds__(THREADS, 1) chain_kernel(const __grid_constant__ Maps M, const Params P) {
  using L = Lay<D>;
  using G = Geo<D>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + L::OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + L::OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L::OFF_BAR + 392);
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
  const int u0 = P.u0, units = G::UNITS - u0;

  int xs = 0, gs = 0, parts = 0, ss = 0;
  if (w == W_LOAD) {
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      if (n >= 2) WAIT(B_XFREE + (n & 1), (uint32_t)(n >> 1) - 1u, 130);
      if (n >= 1) WAIT(B_GFREE, (uint32_t)n - 1u, 131);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_GFULL], 2 * LT);
        for (int m = 0; m < 2; ++m) {
          if (DK) tma_load_4d(sm + L::OFF_G + m * LT, &M.y, &bars[B_GFULL], 0, k.tok + m * 128, k.h, k.b);
          else tma_load_4d(sm + L::OFF_G + m * LT, &M.y, &bars[B_GFULL], 0, k.tok + m * 128, k.head, 0);   // dO': dense over all heads
        }
        uint64_t* bar = &bars[B_XFULL + (n & 1)];
        mbar_arrive_expect_tx(bar, 2 * LT);
        for (int m = 0; m < 2; ++m) tma_load_4d(sm + ((n & 1) * 2 + m) * LT, &M.x, bar, 0, k.tok + m * 128, k.h, k.b);
      }
      xs = gs = n + 1;
      const uint8_t* src = P.S + ((long long)k.st * G::UNITS + u0) * G::UNIT_BYTES;
      for (int j = 0; j < units; ++j, ++ss) {
        const int s = ss % S_STAGES;
        if (ss >= S_STAGES) WAIT(B_SEMPTY + s, (uint32_t)(ss / S_STAGES) - 1u, 132);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&bars[B_SFULL + s], G::UNIT_BYTES);
          bulk_load(sm + L::OFF_S + s * G::UNIT_BYTES, src + (long long)j * G::UNIT_BYTES, G::UNIT_BYTES, &bars[B_SFULL + s]);
        }
      }
      if (P.part) {
        if (n >= 1) WAIT(B_PFREE, (uint32_t)n - 1u, 133);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&bars[B_PFULL], 2 * (D / 32) * LT);
          for (int m = 0; m < 2; ++m)
            for (int c = 0; c < D / 32; ++c)
              tma_load_4d(sm + L::OFF_P + (m * (D / 32) + c) * LT, &M.part, &bars[B_PFULL], 32 * c, k.tok + m * 128, k.head, 0);
        }
        parts = n + 1;
      }
    }
  } else if (w < 2) {
    constexpr uint32_t ID = make_idesc_bf16(128, 64, 0, 0);
    const uint32_t g = tmem + 64u * w;
    uint32_t sg = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      WAIT(B_GT + w, (uint32_t)n, 134);
      for (int j = 0; j < units; ++j, ++sg) {
        const uint32_t s = sg % S_STAGES, buf = sg & 1u;
        WAIT(B_SFULL + (int)s, sg / S_STAGES, 135);
        if (sg >= 2) WAIT(B_DFREE + 2 * w + (int)buf, (sg >> 1) - 1u, 136);
        tc_fence_after_sync();
        const uint64_t dS = make_smem_desc(smem_u32(sm + L::OFF_S) + s * G::UNIT_BYTES, 1024, 128, 0);
#pragma unroll
        for (int kk = 0; kk < (D + 16) / 16; ++kk)
          mma_ts_elect(tmem + COL_D + 128u * w + 64u * buf, g + 8u * kk, dS + (uint64_t)(128 * kk), ID, kk > 0 ? 1u : 0u);
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
    uint32_t sg = 0;
    int n = 0;
    for (int idx = blockIdx.x; idx < P.nitems && *abort_flag == 0; idx += gridDim.x, ++n) {
      const Work k = work(idx, P);
      const int row = k.tok + m * 128 + l;
      WAIT(B_GFULL, (uint32_t)n, 137);
      {
        const uint8_t* src = sm + L::OFF_G + m * LT;
        uint32_t r[D / 2], r8[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
        for (int c = 0; c < D / 8; ++c) {
          const uint4 v = sw_chunk(src, l, c);
          r[4 * c] = v.x; r[4 * c + 1] = v.y; r[4 * c + 2] = v.z; r[4 * c + 3] = v.w;
        }
        pair::tmem_st<D / 2>(lane_addr + 64u * m, r);
        // one, or -delta (a bf16 number, see prologue_kernel)
        r8[0] = DK ? 0x00003F80u : bf16x2(row < P.n ? __ldg(P.ndelta + (long long)k.head * P.nd_ld + row) : 0.f, 0.f);
        tmem_st8(lane_addr + 64u * m + D / 2, r8);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars[B_GT + m]);
          mbar_arrive(&bars[B_GFREE]);
        }
      }
      WAIT(B_XFULL + (n & 1), (uint32_t)(n >> 1), 138);
      const uint8_t* x = sm + ((n & 1) * 2 + m) * LT;
      uint64_t acc[D / 2];
#pragma unroll
      for (int i = 0; i < D / 2; ++i) acc[i] = 0ull;
      // the eight values of block c of this token's row, in pairs
      auto block = [&](int c, uint64_t (&v)[4]) {
        const uint4 q = sw_chunk(x, l, c);
        v[0] = pack2u(q.x << 16, q.x & 0xffff0000u); v[1] = pack2u(q.y << 16, q.y & 0xffff0000u);
        v[2] = pack2u(q.z << 16, q.z & 0xffff0000u); v[3] = pack2u(q.w << 16, q.w & 0xffff0000u);
      };
      auto next_unit = [&]() -> uint32_t {   // waits for the unit's dphi; its TMEM address
        const uint32_t buf = sg & 1u;
        WAIT(B_D + 2 * m + (int)buf, sg >> 1, 139);
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
        for (int a = 0; a < G::NB; ++a) {
          uint64_t xa[4], t[8];
          block(a, xa);
#pragma unroll
          for (int i = 0; i < 8; ++i) t[i] = 0ull;
#pragma unroll
          for (int b = a; b < G::NB; ++b) {
            uint64_t xb[4];
            if (b == a) { xb[0] = xa[0]; xb[1] = xa[1]; xb[2] = xa[2]; xb[3] = xa[3]; }
            else block(b, xb);
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
      {   // the linear unit
        const uint32_t addr = next_unit();
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t d[32];
          tmem_ld32(addr + 32u * c, d);
          tmem_ld_wait();
          if (c == D / 32 - 1) unit_done();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[16 * c + j] = add2(acc[16 * c + j], pack2u(d[2 * j], d[2 * j + 1]));
        }
      }
      if (lane == 0) mbar_arrive(&bars[B_XFREE + (n & 1)]);
      uint8_t* own = sm + L::OFF_P + m * (D / 32) * LT + l * 128;
      if (P.part) {
        WAIT(B_PFULL, (uint32_t)n, 140);
#pragma unroll
        for (int q = 0; q < D / 4; ++q) {
          const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(own + (q >> 3) * LT + (((q & 7) ^ sw) << 4));
          acc[2 * q] = add2(acc[2 * q], p.x);
          acc[2 * q + 1] = add2(acc[2 * q + 1], p.y);
        }
      } else if (n > 0) {
        if (lane == 0) bulk_wait_read_all();
        __syncwarp();
      }
#pragma unroll
      for (int q = 0; q < D / 8; ++q)
        *reinterpret_cast<uint4*>(own + ((q ^ sw) << 4)) = make_uint4(bf16x2(acc[4 * q]), bf16x2(acc[4 * q + 1]), bf16x2(acc[4 * q + 2]), bf16x2(acc[4 * q + 3]));
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && row < P.n) {
        tma_store_4d(&M.out, own, 0, row, k.h, k.b);
        bulk_commit_group();
      }
      if (P.part) {
        if (lane == 0) {
          bulk_wait_read_all();
          mbar_arrive(&bars[B_PFREE]);
        }
        __syncwarp();
      }
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

// ---- states of the segments -> weighted bf16 operands of the state before (after) each segment ----------------------------
// raw: float32 [head][ns][rows][D + 4].  Inclusive running sum over the segments (reverse: from the last one), times the
// polynomial weights, rounded once.  total (optional): raw has one segment more, and the sum over all of them is returned in
// float32, unweighted.  A thread owns (unit, row, 8-column block) of a head.
template <int D>
__global__ void __launch_bounds__(64 * (D / 8 + 2)) pack_kernel(const float* __restrict__ raw, uint8_t* __restrict__ S, float* __restrict__ cst, int ns, int reverse,
                                                                int order, float c0, float c1, float c2, float* __restrict__ total) {
  using G = Geo<D>;
  const int u0 = order == 2 ? 0 : G::NPAIR;
  const int u = u0 + blockIdx.x, head = blockIdx.y, r = threadIdx.x & 63, cb = threadIdx.x >> 6;
  const int rows = (order == 2 ? 64 * G::NPAIR : 0) + D + 1;
  const bool lin = u == G::NPAIR;
  float wgt = c1;
  if (!lin) {
    int a, b;
    pair_decode(u, G::NB, a, b);
    wgt = a == b ? c2 : 2.f * c2;
  }
  const bool live = (!lin || r < D) && cb <= D / 8;
  const int nraw = ns + (total != nullptr);
  const float* src = raw + (long long)head * nraw * rows * G::STATE_LD + (long long)(64 * (u - u0) + r) * G::STATE_LD + 8 * cb;
  uint8_t* dst = S + ((long long)head * ns * G::UNITS + u) * G::UNIT_BYTES + cb * 1024 + r * 16;
  const long long src_step = (long long)rows * G::STATE_LD, dst_step = (long long)G::UNITS * G::UNIT_BYTES;
  // the constant row has no place among the features: its weighted sums go to cst
  const bool is_const = lin && r == 0;
  const float* csrc = raw + (long long)head * nraw * src_step + (long long)(rows - 1) * G::STATE_LD + 8 * cb;
  float s[8] = {}, cs[8] = {};
#pragma unroll 4
  for (int i = 0; i < nraw; ++i) {
    const int k = reverse ? nraw - 1 - i : i;
    if (live) {
      const float4 x = *reinterpret_cast<const float4*>(src + k * src_step);
      s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w;
      if (cb < D / 8) {
        const float4 y = *reinterpret_cast<const float4*>(src + k * src_step + 4);
        s[4] += y.x; s[5] += y.y; s[6] += y.z; s[7] += y.w;
      }
    }
    uint4 o;
    if (cb < D / 8) {
      o.x = bf16x2(s[0] * wgt, s[1] * wgt); o.y = bf16x2(s[2] * wgt, s[3] * wgt);
      o.z = bf16x2(s[4] * wgt, s[5] * wgt); o.w = bf16x2(s[6] * wgt, s[7] * wgt);
    } else {
      o = make_uint4(bf16x2(s[0] * wgt, 0.f), 0u, 0u, 0u);
    }
    if (k < ns) *reinterpret_cast<uint4*>(dst + k * dst_step) = o;
    if (is_const && cb <= D / 8) {
      const float4 x = *reinterpret_cast<const float4*>(csrc + k * src_step);
      float* c = cst + ((long long)head * ns + k) * G::CST + 8 * cb;
      cs[0] += x.x; cs[1] += x.y; cs[2] += x.z; cs[3] += x.w;
      if (k < ns) reinterpret_cast<float4*>(c)[0] = make_float4(cs[0] * c0, cs[1] * c0, cs[2] * c0, cs[3] * c0);
      if (cb < D / 8) {
        const float4 y = *reinterpret_cast<const float4*>(csrc + k * src_step + 4);
        cs[4] += y.x; cs[5] += y.y; cs[6] += y.z; cs[7] += y.w;
        if (k < ns) reinterpret_cast<float4*>(c)[1] = make_float4(cs[4] * c0, cs[5] * c0, cs[6] * c0, cs[7] * c0);
      }
    }
  }
  if (total != nullptr && cb <= D / 8) {
    float* t = total + ((long long)head * rows + 64 * (u - u0) + r) * G::STATE_LD + 8 * cb;
    if (live) {
      reinterpret_cast<float4*>(t)[0] = make_float4(s[0], s[1], s[2], s[3]);
      if (cb < D / 8) reinterpret_cast<float4*>(t)[1] = make_float4(s[4], s[5], s[6], s[7]);
    }
    if (is_const) {
      t = total + ((long long)head * rows + rows - 1) * G::STATE_LD + 8 * cb;
      reinterpret_cast<float4*>(t)[0] = make_float4(cs[0], cs[1], cs[2], cs[3]);
      if (cb < D / 8) reinterpret_cast<float4*>(t)[1] = make_float4(cs[4], cs[5], cs[6], cs[7]);
    }
  }
}

#include "long_f32.cuh"

}  // namespace lng
