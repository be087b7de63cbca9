// Pairwise tcgen05 / TMEM kernels: the scores are evaluated tile by tile and nothing is carried between tiles, so
//     forward   S = Q K^T,             P = f(S),                                  O' = P V,  g = row sums of P
//     dq        S = Q K^T, dP = dO' V^T, dS = f'(S) (dP - delta),                 dq = dS K
//     dk, dv    the transposes with a key tile held:                              dv = P^T dO',  dk = dS^T Q
// where dO' = dO / g and delta = (dO . o) / g.  Cost is quadratic in the length, 14 d products per visible pair against
// 2145 x 65 products per token and moment pass at d = 64: below several thousand tokens this is the smaller number, every
// thread block is independent (no scan over the sequence, no partial sums in memory), and each result is written once,
// in its own type.  pair_takes_* hold the rule that chooses between this and the moment scans.
//
// A work item holds 128 rows (256 in the forward: two tiles that take turns on the tensor pipe; keys for dk / dv, queries
// otherwise) and streams 128-row tiles of the other side through a TMA ring.  Scores land in TMEM as [held x streamed];
// the element-wise warps turn them into the bf16 A operand of the second product in place, and the streamed tile is read
// from shared memory K-major by the first product and MN-major by the second: nothing is transposed or copied.
//
// One thread block per SM works through items.  A block asks the hardware scheduler for its next item (cluster launch
// control: it takes over a block that has not started), so the items' lengths may differ by any factor; the loads and
// first products of the next item run under the last tiles and the stores of the current one.
//
// Bound by no pipe alone, and where the GPU is busy for long, by power.  ncu (forward, dk / dv, dq), 64 heads of 4096 x 64: tensor
// pipe active in 67, 69, 70 % of the clocks, issue slots 47, 61, 38 %; 128 heads of 2048 x 32: 33, 35, 40 % and 46, 65, 57 %.  128 heads
// of 4096 x 64 back to back draw 1000 W and run at 1.55 to 1.65 GHz (1.23 ms for forward and backward, 1.07 at 1.9 GHz).  Measured (us,
// forward and backward; the scans of the moment engine before): 128 heads of 4096 x 64, causal 2930 -> 1070; of 1024 x 64 570 -> 114;
// of 2048 x 32 1533 -> 255.  Heads of 16 dims have the kernels of pair_f32.cuh.
#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "launchers.cuh"
#include "pair_launchers.cuh"
#include "tc_launchers.cuh"
#include "tc_phi.cuh"
#include "tc_ptx.cuh"

namespace fm {
namespace pair {

using namespace tc;

__device__ int g_status = 0;
__device__ int g_wait_hist[256];

constexpr long long WAIT_CYCLES = 4000000000ll;   // ~2 s at 2 GHz
constexpr int R = 128;                  // held rows of one accumulator (the TMEM lanes)
constexpr int T = 128;                  // streamed rows per tile
constexpr int W_SCORE = 0, W_ACC = 1, W_LOAD = 2, W_EW = 4;   // warp roles: two issuers, loader, (spare), element-wise warps
constexpr int X_BYTES = T * 128;        // operand tile: 128-byte rows whatever the head dim (narrow heads zero-filled by the copy engine)
constexpr int STAGES = 4;               // ring of streamed tile pairs
enum Kind { FWD = 0, DQ = 1, DKV = 2 };
// Element-wise warps: sixteen, four per TMEM lane quarter (32 columns each), in the backward kernels.  A tile is a chain of waits and
// TMEM accesses around some hundred instructions; with two warps per scheduler nothing ran beside it for half of the time.  Eight ->
// sixteen (us): 128 heads of 2048 x 32 dq 84 -> 79, dk / dv 124 -> 111; 192 of 577 x 64 without a mask dk / dv 47 -> 44.  dq with 64
// dims has three operations per score and keeps eight: 343 with sixteen, 335 with eight (128 heads of 4096).  The forward has eight,
// two per quarter, one per held tile, because a row's weights are added up there: one thread does it, in the order of the columns,
// and every bit of g, which the outputs and gradients are divided by, stays what it is.  us forward, 128 heads of 4096 x 64, of 1024 x
// 64, 192 of 577 x 64, 128 of 2048 x 32: eight 247, 31, 33, 68; sixteen with a row in two parts 247, 31, 31, 62, but other bits; sixteen
// with the same bits: four threads a row (16-lane loads) 261, 32, 33, 67; the chains handed from warp to warp 296, 36, 37, 80.
template <int D, int KIND>
constexpr int EW = KIND == FWD || (KIND == DQ && D == 64) ? 8 : 16;
template <int D, int KIND>
constexpr int THREADS = (W_EW + EW<D, KIND>) * 32;

struct Params {
  View out0, out1;            // FWD: o, g; DQ: dq; DKV: dk, dv
  const float* ndelta;        // [batch*heads][nd_ld]: -delta per query, zero from nq on
  int nd_ld;
  int heads, nr, nx;          // held rows, streamed rows per head
  int off, causal;            // query l sees the keys up to l + off
  int window;                 // 0, or (causal, off = 0): only the keys of the query's own window of this many tokens
  int part_lo, part_hi;       // rows whose results are partial: float32 into `part` (Maps::p0, p1), not divided
  int ntiles;                 // items per head
  int group, last, ngroups;   // heads per group of the item order, and in its last group
  uint32_t mul_g, mul_t, mul_l, mul_h;   // quotients by group * ntiles, group, last and heads without a division: (n * mul) >> shift
  int sh_g, sh_t, sh_l, sh_h;
  int vec0, vec1;             // rows of out0 / out1 start on 16-byte boundaries: written by the copy engine
  float c0, c1, c2;
  float k, w0, w1;            // completed square (see SQ): c0 / c2 - h^2; factors of out0 and out1
  uint32_t h01, h2;           // h = c1 / (2 c2) as the sum of three bf16 numbers
};

// ---- two-lane float32 arithmetic -------------------------------------------------------------------------
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  __nv_bfloat162 r = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2(uint64_t v) {
  float a, b;
  unpack2(v, a, b);
  return bf16x2(a, b);
}

__device__ __noinline__ void fail_record(int code, volatile int* abort_flag) {
  if (*abort_flag == 0) atomicAdd(&g_wait_hist[code & 255], 1);
  *abort_flag = 1;
  atomicExch(&g_status, code);
}
__device__ __noinline__ void wait_slow(uint64_t* bar, uint32_t parity, int code, volatile int* abort_flag) {
  if (*abort_flag == 0 && !mbar_wait_abortable(bar, parity, WAIT_CYCLES, abort_flag)) fail_record(code, abort_flag);
}
// Waits for the phase of parity `parity`.  Returns in any case: when the wait runs out the abort flag is up, every later
// wait of the block falls through at once and the roles run out of items (next_item).  No caller branches on the outcome,
// which keeps the issuer's control flow warp-uniform and its operands in uniform registers.
__device__ __forceinline__ void wait_fast(uint64_t* bar, uint32_t parity, int code, volatile int* abort_flag) {
  if (!mbar_try_wait(bar, parity)) wait_slow(bar, parity, code, abort_flag);
}

// N consecutive TMEM columns of this thread's lane
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t addr, uint32_t (&r)[N]) {
  if constexpr (N == 32) tmem_ld32(addr, r);
  else if constexpr (N == 16) tmem_ld16(addr, r);
  else tmem_ld8(addr, r);
}
template <int N>
__device__ __forceinline__ void tmem_st(uint32_t addr, const uint32_t (&r)[N]) {
  if constexpr (N == 32) tmem_st32(addr, r);
  else if constexpr (N == 16) tmem_st16(addr, r);
  else tmem_st8(addr, r);
}

// ---- cluster launch control: the next block of the grid that has not started, or none ---------------------
__device__ __forceinline__ void clc_try_cancel(void* smem16, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
               ::"r"(smem_u32(smem16)), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ int clc_read(const void* smem16) {   // block index, or -1
  uint32_t ok, x;
  asm volatile(
      "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "mov.b32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=r"(ok), "=r"(x)
      : "r"(smem_u32(smem16))
      : "memory");
  return ok ? (int)x : -1;
}

constexpr int OFF_HELD = 0;                              // two sets of two held tiles
constexpr int OFF_X = 4 * X_BYTES;
constexpr int STAGE = 2 * X_BYTES;
constexpr int OFF_ND = OFF_X + STAGES * STAGE;           // DKV: -delta of the streamed queries, T floats per stage
constexpr int OFF_H = OFF_ND + STAGES * T * 4;              // SQ: two constant 128 x 16 operands whose product is h everywhere
constexpr int OFF_CLC = OFF_H + 2 * R * 32;         // ring of 16-byte answers of the scheduler
constexpr int CLC = 4;
constexpr int OFF_BAR = OFF_CLC + 16 * CLC;
constexpr int SMEM_BYTES = OFF_BAR + 512 + 1024;
static_assert(SMEM_BYTES <= 232448, "shared memory budget");
// barrier slots
constexpr int B_FULL = 0, B_EMPTY = 4, B_HFULL = 8, B_HEMPTY = 10, B_S = 12, B_READS = 14, B_READD = 16, B_P = 17, B_SFREE = 19, B_ACC = 21,
              B_AFREE = 23, B_CFULL = 25, B_CEMPTY = B_CFULL + CLC, B_DRAIN = B_CEMPTY + CLC, B_COUNT = B_DRAIN + 2;
static_assert(B_COUNT * 8 <= 384, "barriers and flags share 512 bytes");
// TMEM columns.  FWD: O' of the two held tiles, their scores, their bf16 tiles P, which have columns of their own: the scores are free
// as soon as they have been read, and the next tile's first products run under this tile's arithmetic.  DQ, DKV: accumulators (dq; dv,
// dk), two score buffers that take turns, dP.  The bf16 A operands of the second products replace the scores that their warp has
// read, 32 columns by 32 columns: no two warps touch the same columns, and a buffer is free again when the second products are
// done.  dP is free as soon as it has been read.
constexpr uint32_t C_ACC = 0, C_ACC1 = 64, C_S = 128, C_DP = 384, C_P = 384;
// where K step kk (16 streamed rows) of P (FWD, DKV) or dS lies
template <int KIND>
__device__ __forceinline__ constexpr uint32_t weights_at(int kk, bool ds) {
  return KIND == FWD ? 8u * kk : 32u * (kk >> 1) + 8u * (kk & 1) + (KIND == DKV && ds ? 16u : 0u);
}

struct Item {
  int head, b, h;
  int r0;          // first held row
  int t0;          // first streamed tile
  int n0, n1;      // streamed tiles of the held tile(s); n1: the second tile of a forward item
};
// The first rows of a causal sequence see few keys: their denominators are small, their gradients a hundred times the rest,
// and what is rounded to bf16 there shows.  Their tile is therefore evaluated without the completed square (below), with the
// roundings of the moment engines, and its denominators sum the rounded weights (the first row's output is then its value).
__device__ __forceinline__ bool first_rows(const Params& P, int r0) { return P.causal && P.off < R && r0 + P.off < R; }

// TILE: streamed rows per tile, HELD: rows of an item
template <int KIND, int TILE, int HELD>
__device__ __forceinline__ Item decode(int idx, const Params& P) {
  // Groups of heads one after the other; within a group the longest items of all its heads first.  Blocks at work share a few
  // heads' streamed tiles in L2 (see order_items), and the last items are short: in the order of the heads, the last head's long
  // items started when everything else was done (64 heads of 4096 tokens: the SMs were idle for 20 % of the forward).
  Item it;
  const int gr = (int)(((uint64_t)(uint32_t)idx * P.mul_g) >> P.sh_g);
  const uint32_t rest = (uint32_t)(idx - gr * P.group * P.ntiles);
  const bool end = gr == P.ngroups - 1;
  const int ti = end ? (int)(((uint64_t)rest * P.mul_l) >> P.sh_l) : (int)(((uint64_t)rest * P.mul_t) >> P.sh_t);
  it.head = gr * P.group + (int)rest - ti * (end ? P.last : P.group);
  it.b = (int)(((uint64_t)(uint32_t)it.head * P.mul_h) >> P.sh_h);
  it.h = it.head - it.b * P.heads;
  it.t0 = 0;
  it.n1 = 0;
  const int all = (P.nx + TILE - 1) / TILE;
  if (KIND == DKV) {
    it.r0 = ti * HELD;
    const int first = it.r0 - P.off;                 // first query that sees key r0
    if (P.causal && first > 0) it.t0 = first / TILE;
    it.n0 = all - it.t0;
    if (P.window) it.n0 = min(it.n0, (it.r0 / P.window + 1) * P.window / TILE - it.t0);
  } else {
    it.r0 = (P.ntiles - 1 - ti) * HELD;
    it.n0 = P.causal ? min(all, (it.r0 + R - 1 + P.off) / TILE + 1) : all;
    if (HELD > R && it.r0 + R < P.nr) it.n1 = P.causal ? min(all, (it.r0 + 2 * R - 1 + P.off) / TILE + 1) : all;
    if (P.window) {   // (a multiple of the item: both tiles are in the same window)
      it.t0 = it.r0 / P.window * (P.window / TILE);
      it.n0 -= it.t0;
      if (it.n1 > 0) it.n1 -= it.t0;
    }
  }
  return it;
}

struct Maps {
  CUtensorMap x, y;     // streamed tiles
  CUtensorMap a, b;     // held tiles
  CUtensorMap o0, o1;   // outputs, 32-row boxes
  CUtensorMap p0, p1;   // partial results in float32, 32-row boxes of 32 columns, dense over all heads
};

template <int D, int KIND, bool SQ>
__global__ void __launch_bounds__(THREADS<D, KIND>, 1) pair_kernel(const __grid_constant__ Maps M, const Params P) {
  constexpr int KS = D / 16;                    // K steps of the first products
  constexpr int HELD_ROWS = KIND == FWD ? 2 * R : R;
  constexpr int EWN = EW<D, KIND>, ROLES = EWN + 3;   // ROLES: warps that follow the items
  constexpr int W = KIND == FWD ? T : 512 / EWN;      // columns of an element-wise warp
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + OFF_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_BAR + 384);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_BAR + 392);
  const int tid = threadIdx.x, lane = tid & 31;
  const int w = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform for the compiler too

  if (tid == 0) {
    for (int i = 0; i < B_COUNT; ++i) {
      uint32_t n = 1;
      if (i >= B_READS && i < B_SFREE) n = KIND == FWD ? EWN / 2 : EWN;           // READS, READD, P
      if (i == B_AFREE || i == B_AFREE + 1) n = KIND == DKV ? 8 : 4;
      if (i == B_HEMPTY || i == B_HEMPTY + 1) n = 1 + (KIND == DQ ? 4 : 8);     // products done, output rows staged there copied
      if (i >= B_CEMPTY && i < B_CEMPTY + CLC) n = ROLES;                       // every role has read the answer
      mbar_init(&bars[i], n);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (SQ && tid < 2 * R) {   // K-major without swizzle: 8 x 8 core matrices of 128 bytes, two along K
    uint8_t* dst = sm + OFF_H + (tid >> 7) * (R * 32) + ((tid & 127) >> 3) * 256 + (tid & 7) * 16;
    *reinterpret_cast<uint4*>(dst) = tid < R ? make_uint4(P.h01, P.h2, 0u, 0u) : make_uint4(0x3F803F80u, 0x00003F80u, 0u, 0u);
    *reinterpret_cast<uint4*>(dst + 128) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
  }
  if (w == W_ACC) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_wait();
  grid_trigger();
  auto WAIT = [&](int bar, uint32_t phase, int code) { wait_fast(&bars[bar], phase & 1u, code, abort_flag); };
  // item n + 1 of this block, for every role: -1 at the end (or when a wait ran out)
  auto next_item = [&](int n) -> int {
    const int c = n & (CLC - 1);
    WAIT(B_CFULL + c, (uint32_t)(n / CLC), 76);
    int idx = *abort_flag != 0 ? -1 : clc_read(sm + OFF_CLC + 16 * c);
    fence_proxy_async_smem();   // the slot is written again by the copy engine's side
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (lane == 0) mbar_arrive(&bars[B_CEMPTY + c]);
    return idx;
  };

  int issued = 0;   // streamed tiles the loader has asked for
  int helds = 0;    // held sets it has asked for
  int asked = 0;    // items it has asked for
  if (w == W_LOAD) {
    // ================= loader and item scheduler =================
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const int c = n & (CLC - 1);
      if (n >= CLC) WAIT(B_CEMPTY + c, (uint32_t)(n / CLC) - 1u, 77);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_CFULL + c], 16);
        clc_try_cancel(sm + OFF_CLC + 16 * c, &bars[B_CFULL + c]);
      }
      asked = n + 1;
      const Item it = decode<KIND, T, HELD_ROWS>(idx, P);
      const int tiles = it.n0 > it.n1 ? it.n0 : it.n1;
      if (n >= 2) WAIT(B_HEMPTY + (n & 1), (uint32_t)(n >> 1) - 1u, 78);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        uint8_t* hs = sm + OFF_HELD + (n & 1) * STAGE;
        uint64_t* bar = &bars[B_HFULL + (n & 1)];
        const bool two = KIND != FWD || it.n1 > 0;
        mbar_arrive_expect_tx(bar, two ? 2 * X_BYTES : X_BYTES);
        tma_load_4d(hs, &M.a, bar, 0, it.r0, it.h, it.b);
        if (KIND == FWD && two) tma_load_4d(hs + X_BYTES, &M.a, bar, 0, it.r0 + R, it.h, it.b);
        if (KIND == DQ) tma_load_4d(hs + X_BYTES, &M.b, bar, 0, it.r0, it.head, 0);   // dO': a dense array over all heads
        if (KIND == DKV) tma_load_4d(hs + X_BYTES, &M.b, bar, 0, it.r0, it.h, it.b);
      }
      helds = n + 1;
      for (int i = 0; i < tiles; ++i) {
        const int s = issued & (STAGES - 1);
        if (issued >= STAGES) WAIT(B_EMPTY + s, (uint32_t)(issued / STAGES) - 1u, 70);
        if (*abort_flag != 0) break;
        if (lane == 0) {
          uint8_t* x = sm + OFF_X + s * STAGE;
          const int row = (it.t0 + i) * T;
          mbar_arrive_expect_tx(&bars[B_FULL + s], 2 * X_BYTES + (KIND == DKV ? T * 4 : 0));
          tma_load_4d(x, &M.x, &bars[B_FULL + s], 0, row, it.h, it.b);
          if (KIND == DKV) {
            tma_load_4d(x + X_BYTES, &M.y, &bars[B_FULL + s], 0, row, it.head, 0);
            bulk_load(sm + OFF_ND + s * T * 4, P.ndelta + (long long)it.head * P.nd_ld + row, T * 4, &bars[B_FULL + s]);
          } else {
            tma_load_4d(x + X_BYTES, &M.y, &bars[B_FULL + s], 0, row, it.h, it.b);
          }
        }
        ++issued;
      }
      idx = next_item(n);
    }
  } else if (w == W_SCORE) {
    // ================= issuer of the first products =================
    // Two issuers, because a wait costs an issuing warp 150 clocks and a tile has up to four of them: one warp's serial
    // chain (1010 clocks per tile in the forward) was twice the tensor pipe's time.
    constexpr uint32_t ID_S = make_idesc_bf16(R, T, 0, 0);
    const uint64_t dHeld = make_smem_desc(smem_u32(sm + OFF_HELD), 16, 1024, 2);
    const uint64_t dXk = make_smem_desc(smem_u32(sm + OFF_X), 16, 1024, 2);          // streamed tile, K-major
    const uint64_t dHa = make_smem_desc(smem_u32(sm + OFF_H), 128, 256, 0), dHb = make_smem_desc(smem_u32(sm + OFF_H + R * 32), 128, 256, 0);
    uint32_t tile = 0;            // streamed tiles so far
    uint32_t cnt[2] = {0, 0};     // FWD: of each held tile
    uint32_t buf = 0, use = 0;    // else: score buffer, times that it has been used
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const Item it = decode<KIND, T, HELD_ROWS>(idx, P);
      const int tiles = it.n0 > it.n1 ? it.n0 : it.n1;
      WAIT(B_HFULL + (n & 1), (uint32_t)(n >> 1), 71);
      const uint64_t dH = dHeld + (uint64_t)((n & 1) * (STAGE >> 4));
      for (int i = 0; i < tiles; ++i) {
        const uint32_t s = tile & (STAGES - 1);
        WAIT(B_FULL + s, tile / STAGES, 73);
        const uint64_t dX = dXk + (uint64_t)(s * (STAGE >> 4)), dY = dX + (X_BYTES >> 4);
#pragma unroll
        for (int m = 0; m < (KIND == FWD ? 2 : 1); ++m) {
          if (i < (m ? it.n1 : it.n0)) {
            if (KIND == FWD) {
              buf = (uint32_t)m;
              if (cnt[m] > 0) WAIT(B_READS + m, cnt[m] - 1u, 80);      // the last scores have been read
              cnt[m]++;
            } else if (use > 0) {
              WAIT(B_SFREE + (int)buf, use - 1u, 80);                  // the second products that read this buffer are done
            }
            tc_fence_after_sync();
            const uint32_t c = tmem + C_S + buf * 128u;
            const bool add_h = SQ && !first_rows(P, it.r0 + m * R);
            if (add_h) mma_ss_elect(c, dHa, dHb, ID_S, 0u);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
              mma_ss_elect(c, dH + (uint64_t)(m * (X_BYTES >> 4) + 2 * ks), dX + (uint64_t)(2 * ks), ID_S, (add_h || ks > 0) ? 1u : 0u);
            if (KIND != FWD) {
              if (tile > 0) WAIT(B_READD, tile - 1u, 82);
              tc_fence_after_sync();
#pragma unroll
              for (int ks = 0; ks < KS; ++ks)
                mma_ss_elect(tmem + C_DP, dH + (uint64_t)((X_BYTES >> 4) + 2 * ks), dY + (uint64_t)(2 * ks), ID_S, ks > 0);
            }
            mma_commit_elect(&bars[B_S + (int)buf]);
            if (KIND != FWD && ++buf == 2) { buf = 0; ++use; }
          }
        }
        ++tile;
      }
      mma_commit_elect(&bars[B_HEMPTY + (n & 1)]);
      idx = next_item(n);
    }
    if (*abort_flag != 0) {   // a wait ran out: leave only after the products in flight
      mma_commit_elect(&bars[B_DRAIN]);
      mbar_wait_bounded(&bars[B_DRAIN], 0, WAIT_CYCLES);
    }
  } else if (w == W_ACC) {
    // ================= issuer of the second products =================
    constexpr uint32_t ID_ACC = make_idesc_bf16(R, D, 0, 1);
    const uint64_t dXm = make_smem_desc(smem_u32(sm + OFF_X), X_BYTES, 1024, 2);     // streamed tile, MN-major
    uint32_t tile = 0, cnt[2] = {0, 0}, buf = 0, use = 0;   // as above
    uint32_t nfree[2] = {0, 0};   // items that have started on each accumulator
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const Item it = decode<KIND, T, HELD_ROWS>(idx, P);
      const int tiles = it.n0 > it.n1 ? it.n0 : it.n1;
      for (int i = 0; i < tiles; ++i) {
        const uint32_t s = tile & (STAGES - 1);
        const uint64_t dX = dXm + (uint64_t)(s * (STAGE >> 4)), dY = dX + (X_BYTES >> 4);
#pragma unroll
        for (int m = 0; m < (KIND == FWD ? 2 : 1); ++m) {
          const int nm = m ? it.n1 : it.n0;
          if (i < nm) {
            if (i == 0) {   // the accumulator's previous rows have been read
              if (nfree[m] > 0) WAIT(B_AFREE + m, nfree[m] - 1u, 79);
              nfree[m]++;
            }
            if (KIND == FWD) { buf = (uint32_t)m; use = cnt[m]++; }
            WAIT(B_P + (int)buf, use, 72);   // the bf16 tiles of the element-wise warps
            tc_fence_after_sync();
            const uint32_t keep = i > 0 ? 1u : 0u;
            const uint32_t a = tmem + (KIND == FWD ? C_P + buf * 64u : C_S + buf * 128u);
#pragma unroll
            for (int kk = 0; kk < T / 16; ++kk)
              mma_ts_elect(tmem + C_ACC + 64u * m, a + weights_at<KIND>(kk, false), (KIND == DQ ? dX : dY) + (uint64_t)(128 * kk), ID_ACC, kk > 0 ? 1u : keep);
            if (KIND == DKV) {
#pragma unroll
              for (int kk = 0; kk < T / 16; ++kk)
                mma_ts_elect(tmem + C_ACC1, a + weights_at<KIND>(kk, true), dX + (uint64_t)(128 * kk), ID_ACC, kk > 0 ? 1u : keep);
            }
            mma_commit_elect(&bars[B_SFREE + (int)buf]);
            if (KIND != FWD && ++buf == 2) { buf = 0; ++use; }
            if (KIND != FWD || m == 1 || i >= it.n1) mma_commit_elect(&bars[B_EMPTY + s]);
            if (i == nm - 1) mma_commit_elect(&bars[B_ACC + m]);
          }
        }
        ++tile;
      }
      idx = next_item(n);
    }
    if (*abort_flag != 0) {
      mma_commit_elect(&bars[B_DRAIN + 1]);
      mbar_wait_bounded(&bars[B_DRAIN + 1], 0, WAIT_CYCLES);
    }
  } else if (w >= W_EW) {
    // ================= element-wise warps =================
    const int we = w - W_EW, quarter = w & 3;
    const int grp = KIND == FWD ? we >> 2 : 0;    // FWD: held tile
    const int part = KIND == FWD ? 0 : we >> 2;   // else: columns of the tile, in quarters or halves
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint64_t C0 = pack2(P.c0, P.c0), C1 = pack2(P.c1, P.c1), C2 = pack2(P.c2, P.c2), C22 = pack2(2.f * P.c2, 2.f * P.c2),
                   K = pack2(P.k, P.k);   // what a mode does not use is not computed
    // which rows this warp writes out: FWD O' of its tile, DKV dv (part 0) and dk (part 1), DQ dq (part 0)
    const bool writes = part < (KIND == DKV ? 2 : 1);
    uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};   // FWD: four chains, one would serialise the additions
    uint64_t ND = 0ull;                           // DQ: -delta of this row
    uint32_t k = 0;          // tiles of this warp's group so far
    uint32_t buf = KIND == FWD ? (uint32_t)grp : 0u;   // score buffer of the next tile
    uint32_t phases = 0;     // per buffer: the phase that the next scores there complete
    uint32_t done = 0;       // items whose results this warp has written
    // Results of an item are written after the next item's first tile, whose products run meanwhile.
    auto results = [&](int n, const Item& it, float total) {
      const int row = it.r0 + grp * R + quarter * 32 + lane;
      WAIT(B_ACC + grp, done, 75);
      ++done;
      tc_fence_after_sync();
      constexpr int CH = 32;
      uint32_t r[D / CH][CH];
#pragma unroll
      for (int c = 0; c < D / CH; ++c) tmem_ld<CH>(lane_addr + 64u * (KIND == FWD ? grp : part) + (uint32_t)(CH * c), r[c]);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_AFREE + grp]);
      const bool second = KIND == DKV && part == 0;   // dv
      const bool first = first_rows(P, it.r0 + grp * R);
      const float w1 = first ? 1.f : P.w1;
      float wgt = second ? w1 : first ? 1.f : P.w0;
      const bool partial = row - lane >= P.part_lo && row - lane < P.part_hi;   // (bounds are multiples of a window)
      if (KIND == FWD && partial) wgt = w1;
      else if (KIND == FWD) wgt = 1.f / total;   // the sum and the products carry the same factor
      if (KIND == FWD) {
        if (row < P.nr)
          reinterpret_cast<float*>(const_cast<void*>(P.out1.ptr))[(long long)it.b * P.out1.sb + (long long)it.h * P.out1.sh + (long long)row * P.out1.sn] = total * w1;
      }
      if (partial) {
        uint8_t* stage = sm + OFF_HELD + (n & 1) * STAGE + (KIND == FWD ? grp : part) * X_BYTES + quarter * 4096;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          if (c > 0) {   // one box of space per warp
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
          }
#pragma unroll
          for (int q = 0; q < CH / 4; ++q)
            *reinterpret_cast<float4*>(stage + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                make_float4(__uint_as_float(r[c][4 * q]) * wgt, __uint_as_float(r[c][4 * q + 1]) * wgt, __uint_as_float(r[c][4 * q + 2]) * wgt,
                            __uint_as_float(r[c][4 * q + 3]) * wgt);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && row < P.nr) {
            tma_store_4d(second ? &M.p1 : &M.p0, stage, 32 * c, row, it.head, 0);
            bulk_commit_group();
          }
        }
      } else if (second ? P.vec1 : P.vec0) {
        // rows -> the item's held set (its products are done), 128-byte swizzle -> the copy engine, which writes whole lines
        // and clips what lies outside; stored by the threads, 32 lines per instruction, this took 1200 to 3000 clocks
        uint8_t* stage = sm + OFF_HELD + (n & 1) * STAGE + (KIND == FWD ? grp : part) * X_BYTES + quarter * 4096;
#pragma unroll
        for (int c = 0; c < D / 8; ++c) {
          const uint32_t(&x)[CH] = r[8 * c / CH];
          const int o = 8 * c % CH;
          uint4 v;
          v.x = bf16x2(__uint_as_float(x[o]) * wgt, __uint_as_float(x[o + 1]) * wgt);
          v.y = bf16x2(__uint_as_float(x[o + 2]) * wgt, __uint_as_float(x[o + 3]) * wgt);
          v.z = bf16x2(__uint_as_float(x[o + 4]) * wgt, __uint_as_float(x[o + 5]) * wgt);
          v.w = bf16x2(__uint_as_float(x[o + 6]) * wgt, __uint_as_float(x[o + 7]) * wgt);
          *reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) = v;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && row < P.nr) {
          tma_store_4d(second ? &M.o1 : &M.o0, stage, 0, row, it.h, it.b);
          bulk_commit_group();
        }
      } else if (row < P.nr) {
        const View& out = second ? P.out1 : P.out0;
        __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(out.ptr)) + (long long)it.b * out.sb + (long long)it.h * out.sh + (long long)row * out.sn;
#pragma unroll
        for (int c = 0; c < D; ++c) p[c] = __float2bfloat16(__uint_as_float(r[c / CH][c % CH]) * wgt);
      }
    };
    // the held set of item n has been read by the copy engine
    auto give_back = [&](int n) {
      if (lane == 0) {
        bulk_wait_read_all();
        mbar_arrive(&bars[B_HEMPTY + (n & 1)]);
      }
    };
    bool pend = false;   // the last item's results are still to be written
    float total = 0.f;   // FWD: this row's sum of the last item
    Item last{};
    int idx = blockIdx.x, n = 0;
    for (; idx >= 0; ++n) {
      const Item it = decode<KIND, T, HELD_ROWS>(idx, P);
      const int nt = (KIND == FWD && grp) ? it.n1 : it.n0;
      const int row = it.r0 + grp * R + quarter * 32 + lane;
      const bool first = first_rows(P, it.r0 + grp * R);
      float next_total = 0.f;
      if (KIND == DQ) {
        const float nd = row < P.nr ? P.ndelta[(long long)it.head * P.nd_ld + row] : 0.f;
        ND = pack2(nd, nd);
      }
      for (int i = 0; i < nt; ++i, ++k) {
        WAIT(B_S + (int)buf, KIND == FWD ? k : phases >> buf, 74);
        if (KIND != FWD) phases ^= 1u << buf;
        if (KIND == DKV) WAIT(B_FULL + (int)(k & (STAGES - 1)), k / STAGES, 81);
        tc_fence_after_sync();
        const int x0 = (it.t0 + i) * T + part * W;   // streamed row of this warp's first column
        // columns [lo, hi) of this row are visible
        int lo = 0, hi = W;
        if (KIND == DKV) {
          if (P.causal) lo = row - P.off - x0;
        } else {
          if (P.causal) hi = row + P.off - x0 + 1;
          if (KIND == FWD && P.nx - x0 < hi) hi = P.nx - x0;   // rows past the last key would count f(0) in the sum
        }
        const bool whole = __all_sync(0xffffffffu, lo <= 0 && hi >= W);
        const uint32_t sa = lane_addr + C_S + buf * 128u + (uint32_t)(W * part);
        if (KIND == FWD) {
          const uint32_t pa = lane_addr + C_P + 64u * grp;
          if (first) {   // general form, the sum of the rounded weights
            if (k > 0) WAIT(B_SFREE + grp, k - 1u, 83);
            tc_fence_after_sync();
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              uint32_t x32[32], pr[16];
              tmem_ld32(sa + 32u * c, x32);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const uint64_t x = pack2u(x32[2 * j], x32[2 * j + 1]);
                float p0, p1;
                unpack2(fma2(fma2(C2, x, C1), x, C0), p0, p1);
                pr[j] = bf16x2(32 * c + 2 * j < hi ? p0 : 0.f, 32 * c + 2 * j + 1 < hi ? p1 : 0.f);
                sum[j & 3] = add2(sum[j & 3], pack2u(pr[j] << 16, pr[j] & 0xffff0000u));
              }
              tmem_st16(pa + 16u * c, pr);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[B_READS + grp]);
          } else {
            uint32_t s[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(sa + 32u * c, s[c]);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars[B_READS + grp]);
            if (k > 0) WAIT(B_SFREE + grp, k - 1u, 83);   // the last tile's second product has read P
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t pr[16];
              if (whole) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const uint64_t x = pack2u(s[c][2 * j], s[c][2 * j + 1]);
                  const uint64_t p = SQ ? fma2(x, x, K) : fma2(fma2(C2, x, C1), x, C0);
                  sum[j & 3] = add2(sum[j & 3], p);
                  pr[j] = bf16x2(p);
                }
              } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const uint64_t x = pack2u(s[c][2 * j], s[c][2 * j + 1]);
                  float p0, p1;
                  unpack2(SQ ? fma2(x, x, K) : fma2(fma2(C2, x, C1), x, C0), p0, p1);
                  if (32 * c + 2 * j >= hi) p0 = 0.f;
                  if (32 * c + 2 * j + 1 >= hi) p1 = 0.f;
                  sum[j & 3] = add2(sum[j & 3], pack2(p0, p1));
                  pr[j] = bf16x2(p0, p1);
                }
              }
              tmem_st16(pa + 16u * c, pr);
            }
          }
          if (i == nt - 1) {
            float a, b;
            unpack2(add2(add2(sum[0], sum[1]), add2(sum[2], sum[3])), a, b);
            sum[0] = sum[1] = sum[2] = sum[3] = 0ull;
            next_total = a + b;
          }
        } else {
          constexpr int CW = W / 32;
          uint32_t d[CW][32], s[CW][32], pr[CW][16], dr[CW][16];
#pragma unroll
          for (int c = 0; c < CW; ++c) {
            tmem_ld32(lane_addr + C_DP + (uint32_t)(W * part + 32 * c), d[c]);
            tmem_ld32(sa + 32u * c, s[c]);
          }
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[B_READD]);
          auto weights = [&](auto square) {   // the element-wise part: f and f' (dP - delta), in bf16
            constexpr bool Q = decltype(square)::value;
#pragma unroll
            for (int c = 0; c < CW; ++c) {
              const ulonglong2* ndp = reinterpret_cast<const ulonglong2*>(sm + OFF_ND + ((k & (STAGES - 1)) * T + W * part + 32 * c) * 4);
#pragma unroll
              for (int j2 = 0; j2 < 8; ++j2) {
                ulonglong2 n2;
                n2.x = n2.y = ND;
                if (KIND == DKV) n2 = ndp[j2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int j = 2 * j2 + e;
                  const uint64_t x = pack2u(s[c][2 * j], s[c][2 * j + 1]);
                  const uint64_t dp = add2(pack2u(d[c][2 * j], d[c][2 * j + 1]), e ? n2.y : n2.x);
                  const uint64_t u = Q ? x : fma2(C22, x, C1);
                  dr[c][j] = bf16x2(mul2(u, dp));
                  if (KIND == DKV) pr[c][j] = bf16x2(Q ? fma2(u, u, K) : fma2(fma2(C2, x, C1), x, C0));
                }
              }
            }
          };
          if (SQ && !first) weights(std::true_type{});
          else weights(std::false_type{});
          if (!whole) {
#pragma unroll
            for (int j = 0; j < W / 2; ++j) {
              const uint32_t keep = ((2 * j >= lo && 2 * j < hi) ? 0x0000ffffu : 0u) | ((2 * j + 1 >= lo && 2 * j + 1 < hi) ? 0xffff0000u : 0u);
              dr[j >> 4][j & 15] &= keep;
              if (KIND == DKV) pr[j >> 4][j & 15] &= keep;
            }
          }
#pragma unroll
          for (int c = 0; c < CW; ++c) {
            if (KIND == DKV) tmem_st16(sa + 32u * c, pr[c]);
            tmem_st16(sa + 32u * c + (KIND == DKV ? 16u : 0u), dr[c]);
          }
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[B_P + (int)buf]);
        if (KIND != FWD) buf ^= 1u;
        if (i == 0 && pend) results(n - 1, last, total);
        if (i == 1 && pend) give_back(n - 1);
      }
      if (nt == 0) {   // FWD, second tile absent: the last item's results now, nothing to stage for this one
        if (pend) {
          results(n - 1, last, total);
          give_back(n - 1);
        }
        if (writes) {
          WAIT(B_HFULL + (n & 1), (uint32_t)(n >> 1), 84);   // (not before the set's last phase is over)
          if (lane == 0) mbar_arrive(&bars[B_HEMPTY + (n & 1)]);
        }
      } else if (nt == 1 && pend) {
        give_back(n - 1);
      }
      pend = writes && nt > 0;
      last = it;
      total = next_total;
      idx = next_item(n);
    }
    if (pend) results(n - 1, last, total);
    if (lane == 0) bulk_wait_read_all();   // before the block's shared memory goes
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {   // a wait ran out: copies in flight still land in this block's shared memory
    if (w == W_LOAD) {
      for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i)
        mbar_wait_bounded(&bars[B_FULL + (i & (STAGES - 1))], (uint32_t)(i / STAGES) & 1u, WAIT_CYCLES);
      for (int i = helds > 2 ? helds - 2 : 0; i < helds; ++i) mbar_wait_bounded(&bars[B_HFULL + (i & 1)], (uint32_t)(i >> 1) & 1u, WAIT_CYCLES);
      for (int i = asked > CLC ? asked - CLC : 0; i < asked; ++i)
        mbar_wait_bounded(&bars[B_CFULL + (i & (CLC - 1))], (uint32_t)(i / CLC) & 1u, WAIT_CYCLES);
    }
    __syncthreads();
  }
  if (w == W_ACC) tmem_dealloc(tmem, 512);
}

// dO' = dO / g in bf16 (dense [batch*heads][nq][ld], ld = D or D + 16) and -delta = -(dO . o) / g, rounded to bf16 as everywhere (zero from nq on).  D / 8 threads per row,
// 16-byte accesses (VEC) or element by element for views that do not allow them.
template <int D, bool VEC>
__global__ void __launch_bounds__(256) prologue_kernel(View dout, View o, View g, __nv_bfloat16* __restrict__ dop, float* __restrict__ ndelta,
                                                       int nq, int nd_ld, int heads, int ld) {
  constexpr int TPR = D / 8;
  grid_wait();
  grid_trigger();
  const int head = blockIdx.y, b = head / heads, h = head - b * heads;
  const int row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, c = (threadIdx.x % TPR) * 8;
  float dv[8], dot = 0.f;
  float inv = 0.f;
  if (row < nq) {
    const __nv_bfloat16* pd = reinterpret_cast<const __nv_bfloat16*>(dout.ptr) + (long long)b * dout.sb + (long long)h * dout.sh + (long long)row * dout.sn + c;
    const __nv_bfloat16* po = reinterpret_cast<const __nv_bfloat16*>(o.ptr) + (long long)b * o.sb + (long long)h * o.sh + (long long)row * o.sn + c;
    inv = 1.f / reinterpret_cast<const float*>(g.ptr)[(long long)b * g.sb + (long long)h * g.sh + (long long)row * g.sn];
    __nv_bfloat16 xd[8], xo[8];
    if (VEC) {
      *reinterpret_cast<uint4*>(xd) = *reinterpret_cast<const uint4*>(pd);
      *reinterpret_cast<uint4*>(xo) = *reinterpret_cast<const uint4*>(po);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) { xd[i] = pd[i]; xo[i] = po[i]; }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      dv[i] = __bfloat162float(xd[i]) * inv;
      dot += dv[i] * __bfloat162float(xo[i]);
    }
  }
#pragma unroll
  for (int m = TPR / 2; m > 0; m >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, m);
  if (row < nq) {
    uint4 r;
    r.x = bf16x2(dv[0], dv[1]); r.y = bf16x2(dv[2], dv[3]); r.z = bf16x2(dv[4], dv[5]); r.w = bf16x2(dv[6], dv[7]);
    __nv_bfloat16* out = dop + ((long long)head * nq + row) * ld;
    *reinterpret_cast<uint4*>(out + c) = r;
    if (c == 0 && ld > D) {   // rows of D + 16 columns: -delta and zeros behind the values
      *reinterpret_cast<uint4*>(out + D) = make_uint4(bf16x2(-dot, 0.f), 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(out + D + 8) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (c == 0 && row < nd_ld) ndelta[(long long)head * nd_ld + row] = row < nq ? __bfloat162float(__float2bfloat16(-dot)) : 0.f;
}

#include "pair_f32.cuh"

}  // namespace pair

#include "long_kernels.cuh"

// ------------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------------
namespace {

// n / d = (n * mul) >> shift for every n < 2^31
void quotient(int d, uint32_t& mul, int& shift) {
  int log = 0;
  while ((1ll << log) < d) ++log;
  shift = 31 + log;
  mul = (uint32_t)(((1ull << shift) + d - 1) / d);
}

template <int D, int KIND, bool SQ>
cudaError_t launch(const pair::Maps& M, const pair::Params& P, int bh, cudaStream_t st) {
  auto kernel = pair::pair_kernel<D, KIND, SQ>;
  static std::atomic<bool> done[64];   // the attribute sticks to the kernel on its device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pair::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
  }
  return launch_after(kernel, dim3((unsigned)(P.ntiles * bh)), pair::THREADS<D, KIND>, pair::SMEM_BYTES, st, M, P);
}
// Heads per group of the item order (decode).  With a mask, items differ in length: as many heads as have their streamed tiles in
// 32 MB (pieces: 64 MB) of L2.  us forward / dq / dk, dv for 16, 32, 64, 128 MB: 128 heads of 4096 x 64 252 / 337 / 453,
// 245 / 337 / 452, 248 / 342 / 457, 273 / 395 / 518; of 1024 x 64 34 / 39 / 48, then 31 / 37 / 47; float32, of 1024 x 64
// 120 / 144 / 198, 113 / 138 / 190, 110 / 135 / 185, 111 / 136 / 189 (few items per block: the last group's long ones decide).
// Without a mask (and within windows) the items are alike, and the order of the heads is best for L2.
void order_items(int d, int es, pair::Params& P, int bh) {
  long long group = 1;
  if (P.causal && !P.window) {
    group = ((es > 2 ? 64ll : 32ll) << 20) / ((long long)P.nx * d * 2 * es);
    group = group < 1 ? 1 : group > bh ? bh : group;
    const long long n = (bh + group - 1) / group;
    group = (bh + n - 1) / n;
  }
  P.group = (int)group;
  P.ngroups = (bh + P.group - 1) / P.group;
  P.last = bh - (P.ngroups - 1) * P.group;
  quotient(P.group * P.ntiles, P.mul_g, P.sh_g);
  quotient(P.group, P.mul_t, P.sh_t);
  quotient(P.last, P.mul_l, P.sh_l);
  quotient(P.heads, P.mul_h, P.sh_h);
}
template <int KIND, bool SQ>
cudaError_t launch_d(int d, const pair::Maps& M, pair::Params& P, int bh, cudaStream_t st) {
  order_items(d, 2, P, bh);
  switch (d) {
    case 32: return launch<32, KIND, SQ>(M, P, bh, st);
    default: return launch<64, KIND, SQ>(M, P, bh, st);
  }
}

View view_of(const fastmax_tensor& t) { return View{t.ptr, t.stride_b, t.stride_h, t.stride_n}; }
bool rows16(const fastmax_tensor& t) {   // every row of a bf16 view starts on a 16-byte boundary
  return ((uintptr_t)t.ptr & 15) == 0 && (t.stride_b & 7) == 0 && (t.stride_h & 7) == 0 && (t.stride_n & 7) == 0;
}
int tiles(int n, int rows = pair::R) { return (n + rows - 1) / rows; }
int nd_ld(int n) { return (n + pair::T - 1) / pair::T * pair::T; }
size_t up256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace
bool f32_registers_ok();
namespace {
// bf16 heads of 16 dims have no tensor-memory engine beside the pairs: their weights stay float32 there (split into pieces, results
// rounded once) as in the CUDA-core engine.  Relative error of dq, 16 heads of 1024 tokens: 1.7e-3 that way, which is the
// rounding of the result, 3.2e-3 with bf16 weights.
bool float32_weights(const fastmax_problem* pb) { return pb->dtype == FASTMAX_F32 || pb->d == 16; }
// a view the copy engine can read (a stride of a size-1 dimension is never used)
bool mappable(const fastmax_tensor& t, const fastmax_problem* pb, int n) {
  if (pb->dtype == FASTMAX_F32) return t.ptr != nullptr;   // split by ordinary loads
  const int64_t big = (int64_t)1 << 39;
  auto ok = [&](int64_t s, int extent) { return extent == 1 || (s > 0 && s < big && (s & 7) == 0); };
  return t.ptr && ((uintptr_t)t.ptr & 15) == 0 && ok(t.stride_n, n) && ok(t.stride_h, pb->heads) && ok(t.stride_b, pb->batch);
}

// rows of a float32 view as the copy engine reads and writes them
bool rows_f32(const fastmax_tensor& t, const fastmax_problem* pb, int n) {
  const int64_t big = (int64_t)1 << 38;
  auto ok = [&](int64_t s, int extent) { return extent == 1 || (s > 0 && s < big && (s & 3) == 0); };
  return t.ptr && ((uintptr_t)t.ptr & 15) == 0 && ok(t.stride_n, n) && ok(t.stride_h, pb->heads) && ok(t.stride_b, pb->batch);
}
// Which form takes a call.  USE_OUT: output alone; USE_TRAIN: forward and backward of a training call (the states of the forward
// are handed on, so both take the same form); USE_PROMPT: output and final state.
enum Use { USE_OUT, USE_TRAIN, USE_PROMPT };
// The pairwise kernels cost about 1e-6 us per visible pair forward and backward (d = 64; d = 32: 1.2e-6 to 0.9e-6, it is bound by the
// same number of scores), windows and states a time per token.  `per_token`: the keys a token sees on average at which both cost the
// same.  us at 128 heads, forward + backward, pairs / windows:
//   order 2, mask:    d = 64 6144 tokens 2375 / 2536, 7168 3326 / 3057; d = 32 2048 349 / 492, 3072 690 / 659
//   order 2, no mask: d = 64 2048 519 / 717, 3072 1106 / 989;           d = 32 1024 167 / 195, 1536 324 / 251
//   order 1, mask:    d = 64 1536 256 / 330, 2048 358 / 425;            d = 32 1536 205 / 240, 2048 313 / 312
//   order 1, no mask: d = 64 768 105 / 110, 1024 148 / 130;             d = 32 768 104 / 110, 1024 150 / 111
// and forward alone: order 2, mask, d = 64 8192 874 / 1103, 11264 1628 / 1535, d = 32 4096 269 / 336, 6144 551 / 475; no mask, d = 64
// 4096 448 / 436, d = 32 1536 82 / 81; order 1, mask, d = 64 2048 101 / 140, 3072 198 / 193, d = 32 2048 96 / 106; no mask, d = 32 1024
// 51 / 42.  Prompts (pairs with the moments beside them / windows): order 2, d = 64 4096 479 / 596, 6144 872 / 925, d = 32 2048 302 /
// 182; order 1, d = 64 1024 78 / 85, d = 32 1024 93 / 70.  At 60 heads training calls cross a little later (order 2, mask, d = 64
// 7168 1425 / 1447; d = 32 4096 505 / 496).  The lines stand where the kernels before the present ones crossed: pairs are now the
// faster form somewhat beyond those of order 1 with a mask (up to some 2500 tokens, 2000 with 32 dims) and of prompts of 64 dims (up to
// some 6500), and windows below that of prompts of 32 dims.
double window_line(const fastmax_problem* pb, Use use) {
  const bool wide = pb->d == 64;
  if (pb->order == 2) {
    if (pb->causal) return use == USE_TRAIN ? (wide ? 3600. : 1500.) : use == USE_PROMPT ? (wide ? 2500. : 1150.) : (wide ? 5500. : 2150.);
    return use == USE_TRAIN ? (wide ? 3100. : 1100.) : (wide ? 4600. : 1600.);
  }
  if (pb->causal) return use == USE_TRAIN ? (wide ? 900. : 800.) : use == USE_PROMPT ? 600. : (wide ? 1450. : 1300.);
  return use == USE_TRAIN ? (wide ? 550. : 600.) : (wide ? 800. : 1100.);
}
int chosen(const fastmax_problem* pb, bool backward, Use use) {   // 0: neither, 1: pair by pair, 2: windows and states
  if (!(pb->flags & FASTMAX_FLAG_PAIRWISE) || (pb->flags & FASTMAX_FLAG_NO_TENSOR_CORES)) return 0;
  if (pb->nq <= 0 || pb->nk <= 0) return 0;
  if ((long long)tiles(pb->nq > pb->nk ? pb->nq : pb->nk) * pb->batch * pb->heads >= (1ll << 31)) return 0;
  const double nq = pb->nq, nk = pb->nk;
  const double pairs = pb->causal ? nq * (nk - 0.5 * (nq - 1.0)) : nq * nk;
  const double per_token = pairs / (0.5 * (nq + nk));
  if (pb->dtype == FASTMAX_F32) {
    // against the CUDA-core engine, whose cost per token goes with d^3 (order 2) or d^2, while six piece products on half-empty
    // tiles hardly get cheaper for narrow heads.  us, forward + backward, pairs / engine: order 2, no mask, d = 64 16 heads 12288 tokens
    // 12900 / 22700, d = 32 32 heads 4096 2110 / 2570, 5120 3180 / 2440, d = 16 64 heads 1536 554 / 576, 2048 796 / 742; mask, d = 16 64
    // heads 4096 1540 / 1983; order 1, mask, d = 64 64 heads 4096 2900 / 3710, d = 16 64 heads 1536 291 / 452, 2048 475 / 474; no mask, 64
    // heads, d = 64 1024 544 / 513, 1280 793 / 633, d = 32 768 190 / 174, d = 16 512 89 / 135, 768 151 / 134.
    const double most = pb->order == 2 ? (pb->d == 64 ? 16000.0 : pb->d == 32 ? 5000.0 : 2000.0)
                        : pb->causal   ? (pb->d == 64 ? 2300.0 : pb->d == 32 ? 1050.0 : 900.0)
                                       : (pb->d == 64 ? 1300.0 : pb->d == 32 ? 800.0 : 600.0);
    // d = 32 with a mask: windows and states (us, forward + backward, pairs / windows: order 2 64 heads 1536 tokens 350 / 433, 2048
    // 557 / 554; order 1 128 heads 768 tokens 232 / 268, 1024 351 / 342)
    if (pb->d == 32 && pb->causal && pb->nq == pb->nk && pb->nq < (1 << 30) && f32_registers_ok() && per_token > (pb->order == 2 ? 900. : 450.)) return 2;
    return per_token <= most && f32_registers_ok() ? 1 : 0;
  }
  // order 1 without a mask: one pass over the tensors (p1_forward_kernel), always the cheapest where it fills the GPU
  if (!backward && pb->order == 1 && !pb->causal && pb->d == 64 && (long long)pb->batch * pb->heads >= 64) return 0;
  // d = 16: float32 weights (float32_weights) against the CUDA-core engine; there is no states kernel.  us, forward + backward of 64
  // heads, pairs / engine: order 2, mask, 4096 tokens 1261 / 1973, 6144 2737 / 2639; no mask, 2048 629 / 736, 4096 2420 / 1388; order 1,
  // mask, 2048 357 / 453, 4096 1260 / 888; no mask, 256 81 / 133, 768 124 / 135, 128 heads 1024 336 / 233.
  if (pb->d == 16)
    return per_token <= (pb->order == 2 ? (pb->causal ? 3000.0 : 2300.0) : pb->causal ? 1200.0 : 700.0) && f32_registers_ok() ? 1 : 0;
  if (per_token <= window_line(pb, use)) return 1;
  if (pb->causal && pb->nq != pb->nk) return per_token <= (pb->order == 2 ? 6500.0 : backward ? 1300.0 : 2000.0) ? 1 : 0;
  if ((long long)(pb->nq > pb->nk ? pb->nq : pb->nk) >= (1ll << 30)) return 0;
  return 2;
}
uint32_t bf16_bits(float x) {
  const __nv_bfloat16 v = __float2bfloat16(x);
  return *reinterpret_cast<const uint16_t*>(&v);
}
// Returns whether the kernels run with the square completed (SQ): order 2 with 64 a0 a2 >= a1^2, i.e. h^2 at most sixteen
// times c0 / c2, so that u^2 + k keeps its accuracy (the reference's coefficients: h^2 half of c0 / c2).
bool fill(const fastmax_problem* pb, pair::Params& P) {
  P.heads = pb->heads;
  P.causal = pb->causal;
  P.off = pb->causal ? pb->nk - pb->nq : 0;
  P.c0 = pb->a0;
  P.c1 = pb->a1 * pb->inv_temperature;
  P.c2 = pb->order == 2 ? pb->a2 * pb->inv_temperature * pb->inv_temperature : 0.f;
  P.w0 = P.w1 = 1.f;
  if (pb->order != 2 || !(fabsf(P.c2) >= 1e-30f) || !(64.0 * pb->a0 * pb->a2 >= (double)pb->a1 * pb->a1)) return false;
  const double h = (double)P.c1 / (2.0 * P.c2);
  if (!(fabs(h) < 1e15)) return false;
  double rest = h, sum = 0.0;
  uint32_t piece[3];
  for (int i = 0; i < 3; ++i) {
    piece[i] = bf16_bits((float)rest);
    const uint32_t bits = piece[i] << 16;
    float back;
    memcpy(&back, &bits, 4);
    sum += back;
    rest -= back;
  }
  P.h01 = piece[0] | piece[1] << 16;
  P.h2 = piece[2];
  P.k = (float)((double)P.c0 / P.c2 - sum * sum);
  return true;
}

}  // namespace

static int forward_form(const fastmax_problem* pb, const fastmax_forward_args* a) {
  if (!a->o.ptr || !a->g.ptr || a->state_in) return 0;
  // (key moments before the state: whether they are packed does not depend on it)
  const Use use = a->key_moments_out || a->key_moments_in ? USE_TRAIN : a->state_out ? USE_PROMPT : USE_OUT;
  const int form = chosen(pb, false, use);
  if (form == 0 || !mappable(a->q, pb, pb->nq) || !mappable(a->k, pb, pb->nk) || !mappable(a->v, pb, pb->nk)) return 0;
  if (form == 2 && pb->dtype == FASTMAX_F32)
    return !a->state_out && rows_f32(a->q, pb, pb->nq) && rows_f32(a->k, pb, pb->nk) && rows_f32(a->o, pb, pb->nq) ? 2 : 0;
  if (form == 2) return rows16(a->o) && mappable(a->o, pb, pb->nq) && (!a->state_out || pb->causal) ? 2 : 0;
  return a->state_out ? 0 : 1;
}
static int backward_form(const fastmax_problem* pb, const fastmax_backward_args* a) {
  if (!a->dq.ptr || !a->dk.ptr || !a->dv.ptr || a->state_in || a->dstate_in || a->dstate_out) return 0;
  const int form = chosen(pb, true, USE_TRAIN);
  if (form == 0 || !mappable(a->q, pb, pb->nq) || !mappable(a->k, pb, pb->nk) || !mappable(a->v, pb, pb->nk)) return 0;
  if (form == 2 && pb->dtype == FASTMAX_F32)
    return rows_f32(a->q, pb, pb->nq) && rows_f32(a->k, pb, pb->nk) && rows_f32(a->dq, pb, pb->nq) && rows_f32(a->dk, pb, pb->nk) && rows_f32(a->dv, pb, pb->nk) ? 2 : 0;
  if (form == 2)
    return rows16(a->dq) && rows16(a->dk) && rows16(a->dv) && mappable(a->dq, pb, pb->nq) && mappable(a->dk, pb, pb->nk) && mappable(a->dv, pb, pb->nk) ? 2 : 0;
  return 1;
}
bool pair_takes_forward(const fastmax_problem* pb, const fastmax_forward_args* a) { return forward_form(pb, a) != 0; }
bool pair_takes_backward(const fastmax_problem* pb, const fastmax_backward_args* a) { return backward_form(pb, a) != 0; }

// ---- float32 ------------------------------------------------------------------------------------------------------------
// bf16 pieces [3][batch*heads][n][d] as a tensor map: piece = batch index, head = batch*heads
static size_t pieces_bytes(const fastmax_problem* pb, int n, int ld = 0) { return up256((size_t)3 * pb->batch * pb->heads * n * (ld > 0 ? ld : pb->d) * 2); }
static size_t input_bytes(const fastmax_problem* pb, int n) { return pb->dtype == FASTMAX_F32 ? pieces_bytes(pb, n) : 0; }   // pieces of q, k or v
static size_t long_forward_workspace(const fastmax_problem* pb);
static size_t long_f32_forward_workspace(const fastmax_problem* pb);
static size_t long_f32_backward_workspace(const fastmax_problem* pb);
static size_t long_backward_workspace(const fastmax_problem* pb);
size_t pair_forward_workspace(const fastmax_problem* pb, const fastmax_forward_args* a) {
  if (forward_form(pb, a) == 2) return pb->dtype == FASTMAX_F32 ? long_f32_forward_workspace(pb) : long_forward_workspace(pb);
  return input_bytes(pb, pb->nq) + 2 * input_bytes(pb, pb->nk);
}
size_t pair_backward_workspace(const fastmax_problem* pb, const fastmax_backward_args* a) {
  if (backward_form(pb, a) == 2) return pb->dtype == FASTMAX_F32 ? long_f32_backward_workspace(pb) : long_backward_workspace(pb);
  const size_t bh = (size_t)pb->batch * pb->heads, delta = up256(bh * nd_ld(pb->nq) * sizeof(float));
  if (float32_weights(pb)) return pieces_bytes(pb, pb->nq) + input_bytes(pb, pb->nq) + 2 * input_bytes(pb, pb->nk) + delta;
  return up256(bh * pb->nq * pb->d * 2) + delta;
}

// rows [first, n) of every piece and head; columns past `cols` read as zero
static bool pieces_map(CUtensorMap* m, void* p, const fastmax_problem* pb, int n, int rows, int ld = 0, int cols = 0, int first = 0) {
  const int64_t bh = (int64_t)pb->batch * pb->heads;
  if (ld == 0) ld = pb->d;
  const fastmax_tensor t{(__nv_bfloat16*)p + (int64_t)first * ld, bh * n * ld, (int64_t)n * ld, ld};
  return tc_make_map(m, t, 3, (int)bh, n - first, 64, rows, true, cols > 0 ? cols : pb->d);
}
static cudaError_t launch_split(const fastmax_problem* pb, const pair::f32::SplitArgs& A, int count, cudaStream_t st) {
  int n = A.n[0];
  for (int i = 1; i < count; ++i) n = A.n[i] > n ? A.n[i] : n;
  const int rows = 256 / (pb->d / 8);
  const dim3 grid((unsigned)((n + rows - 1) / rows), (unsigned)(pb->batch * pb->heads), (unsigned)count);
  LaunchScope ls(KK_PAIR_SPLIT, st);
  switch (pb->d) {
    case 16: return launch_after(pair::f32::split_kernel<16>, grid, 256, 0, st, A, pb->heads);
    case 32: return launch_after(pair::f32::split_kernel<32>, grid, 256, 0, st, A, pb->heads);
    default: return launch_after(pair::f32::split_kernel<64>, grid, 256, 0, st, A, pb->heads);
  }
}
template <int D, int KIND, int IN>
static cudaError_t launch_f32(const pair::Maps& M, const pair::Params& P, int bh, cudaStream_t st) {
  auto kernel = pair::f32::pair_f32_kernel<D, KIND, IN>;
  constexpr int bytes = pair::f32::Lay<KIND>::BYTES;
  static std::atomic<bool> done[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
  }
  return launch_after(kernel, dim3((unsigned)(P.ntiles * bh)), pair::f32::THREADS_F<KIND>, bytes, st, M, P);
}
template <int KIND>
static cudaError_t launch_f32_d(const fastmax_problem* pb, const pair::Maps& M, pair::Params& P, cudaStream_t st) {
  const int bh = pb->batch * pb->heads;
  order_items(pb->d, pb->dtype == FASTMAX_F32 ? 6 : 2, P, bh);
  if (pb->dtype == FASTMAX_BF16) return launch_f32<16, KIND, 1>(M, P, bh, st);
  switch (pb->d) {
    case 16: return launch_f32<16, KIND, 3>(M, P, bh, st);
    case 32: return launch_f32<32, KIND, 3>(M, P, bh, st);
    default: return launch_f32<64, KIND, 3>(M, P, bh, st);
  }
}
// dk / dv move registers between their warps (setmaxnreg), which only ends if the blocks are launched with what the budget
// in pair_f32.cuh assumes
bool f32_registers_ok() {
  static const bool ok = [] {
    auto right = [](auto kernel) {
      cudaFuncAttributes a{};
      return cudaFuncGetAttributes(&a, kernel) == cudaSuccess && a.numRegs == pair::f32::REG_LAUNCH;
    };
    return right(pair::f32::pair_f32_kernel<16, pair::DKV, 3>) && right(pair::f32::pair_f32_kernel<32, pair::DKV, 3>) &&
           right(pair::f32::pair_f32_kernel<64, pair::DKV, 3>) && right(pair::f32::pair_f32_kernel<16, pair::DKV, 1>);
  }();
  return ok;
}

// Tensor map of q, k or v: their pieces, or (bf16) the tensor itself
static bool input_map(CUtensorMap* m, const fastmax_tensor& t, void* pieces, const fastmax_problem* pb, int n, int rows) {
  return pb->dtype == FASTMAX_F32 ? pieces_map(m, pieces, pb, n, rows) : tc_make_map(m, t, pb->batch, pb->heads, n, 64, rows, true, pb->d);
}
static cudaError_t split_inputs(const fastmax_problem* pb, const fastmax_tensor& q, const fastmax_tensor& k, const fastmax_tensor& v, void* qp, void* kp, void* vp,
                                cudaStream_t st) {
  if (pb->dtype != FASTMAX_F32) return cudaSuccess;
  return launch_split(pb, pair::f32::SplitArgs{{view_of(q), view_of(k), view_of(v)}, {(__nv_bfloat16*)qp, (__nv_bfloat16*)kp, (__nv_bfloat16*)vp},
                                               {pb->nq, pb->nk, pb->nk}, {pb->d, pb->d, pb->d}}, 3, st);
}
static int pair_f32_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, cudaStream_t st) {
  char* base = (char*)ws;
  void *qp = base, *kp = base + input_bytes(pb, pb->nq), *vp = base + input_bytes(pb, pb->nq) + input_bytes(pb, pb->nk);
  pair::Maps M;
  if (!input_map(&M.a, a->q, qp, pb, pb->nq, pair::R) || !input_map(&M.x, a->k, kp, pb, pb->nk, pair::f32::TF) ||
      !input_map(&M.y, a->v, vp, pb, pb->nk, pair::f32::TF))
    return FASTMAX_ERR_UNSUPPORTED;
  M.b = M.o0 = M.o1 = M.a;
  cudaError_t e = split_inputs(pb, a->q, a->k, a->v, qp, kp, vp, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  pair::Params P{};
  fill(pb, P);
  P.out0 = view_of(a->o);
  P.out1 = view_of(a->g);
  P.nr = pb->nq;
  P.nx = pb->nk;
  P.ntiles = tiles(pb->nq);
  P.vec0 = rows_f32(a->o, pb, pb->nq);
  LaunchScope ls(KK_PAIR_F32_FWD, st);
  e = launch_f32_d<pair::FWD>(pb, M, P, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

template <typename T, int D>
static cudaError_t launch_prologue_f32(const fastmax_problem* pb, const fastmax_backward_args* a, __nv_bfloat16* dop, float* nd, int dld, cudaStream_t st) {
  const int ld = nd_ld(pb->nq), rows = 256 / (D / 8);
  const dim3 grid((unsigned)((ld + rows - 1) / rows), (unsigned)(pb->batch * pb->heads));
  auto vec = [](const fastmax_tensor& t) {
    constexpr int64_t odd = 16 / sizeof(T) - 1;
    return ((uintptr_t)t.ptr & 15) == 0 && (t.stride_b & odd) == 0 && (t.stride_h & odd) == 0 && (t.stride_n & odd) == 0;
  };
  if (vec(a->o) && vec(a->d_out))
    return launch_after(pair::f32::prologue_f32_kernel<T, D, true>, grid, 256, 0, st, view_of(a->d_out), view_of(a->o), view_of(a->g), dop, nd, pb->nq, ld, pb->heads, dld);
  return launch_after(pair::f32::prologue_f32_kernel<T, D, false>, grid, 256, 0, st, view_of(a->d_out), view_of(a->o), view_of(a->g), dop, nd, pb->nq, ld, pb->heads, dld);
}

static int pair_f32_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, cudaStream_t st) {
  const size_t nqb = input_bytes(pb, pb->nq), nkb = input_bytes(pb, pb->nk), dob = pieces_bytes(pb, pb->nq);
  char* base = (char*)ws;
  void *dp = base, *qp = base + dob, *kp = base + dob + nqb, *vp = base + dob + nqb + nkb;
  float* nd = (float*)(base + dob + nqb + 2 * nkb);
  pair::Maps M, N;   // M: dq, N: dk and dv
  if (!input_map(&M.a, a->q, qp, pb, pb->nq, pair::R) || !pieces_map(&M.b, dp, pb, pb->nq, pair::R) ||
      !input_map(&M.x, a->k, kp, pb, pb->nk, pair::f32::TF) || !input_map(&M.y, a->v, vp, pb, pb->nk, pair::f32::TF) ||
      !input_map(&N.a, a->k, kp, pb, pb->nk, pair::R) || !input_map(&N.b, a->v, vp, pb, pb->nk, pair::R) ||
      !input_map(&N.x, a->q, qp, pb, pb->nq, pair::f32::TF) || !pieces_map(&N.y, dp, pb, pb->nq, pair::f32::TF))
    return FASTMAX_ERR_UNSUPPORTED;
  M.o0 = M.o1 = N.o0 = N.o1 = M.a;
  cudaError_t e = split_inputs(pb, a->q, a->k, a->v, qp, kp, vp, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  {
    LaunchScope ls(KK_PROLOGUE, st);
    __nv_bfloat16* dop = (__nv_bfloat16*)dp;
    if (pb->dtype == FASTMAX_BF16) e = launch_prologue_f32<__nv_bfloat16, 16>(pb, a, dop, nd, pb->d, st);
    else if (pb->d == 16) e = launch_prologue_f32<float, 16>(pb, a, dop, nd, pb->d, st);
    else if (pb->d == 32) e = launch_prologue_f32<float, 32>(pb, a, dop, nd, pb->d, st);
    else e = launch_prologue_f32<float, 64>(pb, a, dop, nd, pb->d, st);
  }
  if (e != cudaSuccess) return report_cuda_error(e);
  pair::Params P{};
  fill(pb, P);
  P.ndelta = nd;
  P.nd_ld = nd_ld(pb->nq);
  pair::Params K = P;
  K.out0 = view_of(a->dk);
  K.out1 = view_of(a->dv);
  K.nr = pb->nk;
  K.nx = pb->nq;
  K.ntiles = tiles(pb->nk);
  K.vec0 = rows_f32(a->dk, pb, pb->nk);
  K.vec1 = rows_f32(a->dv, pb, pb->nk);
  {
    LaunchScope ls(KK_PAIR_F32_BWD_KV, st);
    e = launch_f32_d<pair::DKV>(pb, N, K, st);
  }
  if (e != cudaSuccess) return report_cuda_error(e);
  P.out0 = P.out1 = view_of(a->dq);
  P.nr = pb->nq;
  P.nx = pb->nk;
  P.ntiles = tiles(pb->nq);
  P.vec0 = rows_f32(a->dq, pb, pb->nq);
  {
    LaunchScope ls(KK_PAIR_F32_BWD_Q, st);
    e = launch_f32_d<pair::DQ>(pb, M, P, st);
  }
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

// ---- bf16 ---------------------------------------------------------------------------------------------------------------
// 32-row boxes of an output view, one per warp; views the copy engine cannot write are stored element by element
static int out_map(CUtensorMap* m, const fastmax_tensor& t, const fastmax_problem* pb, int n) {
  return rows16(t) && tc_make_map(m, t, pb->batch, pb->heads, n, 64, 32, true, pb->d) ? 1 : 0;
}

template <int D>
static cudaError_t launch_prologue(const fastmax_problem* pb, const fastmax_backward_args* a, __nv_bfloat16* dop, float* nd, int dld, cudaStream_t st) {
  const int ld = nd_ld(pb->nq), rows = 256 / (D / 8);
  const dim3 grid((unsigned)((ld + rows - 1) / rows), (unsigned)(pb->batch * pb->heads));
  if (rows16(a->o) && rows16(a->d_out))
    return launch_after(pair::prologue_kernel<D, true>, grid, 256, 0, st, view_of(a->d_out), view_of(a->o), view_of(a->g), dop, nd, pb->nq, ld, pb->heads, dld);
  return launch_after(pair::prologue_kernel<D, false>, grid, 256, 0, st, view_of(a->d_out), view_of(a->o), view_of(a->g), dop, nd, pb->nq, ld, pb->heads, dld);
}
static cudaError_t launch_prologue_any(const fastmax_problem* pb, const fastmax_backward_args* a, __nv_bfloat16* dop, float* nd, int dld, cudaStream_t st) {
  LaunchScope ls(KK_PROLOGUE, st);
  return pb->d == 32 ? launch_prologue<32>(pb, a, dop, nd, dld, st) : launch_prologue<64>(pb, a, dop, nd, dld, st);
}

// ---- long bf16 sequences (long_kernels.cuh) -----------------------------------------------------------------------------
namespace {

// Window of the pairwise part: its cost grows with the window, what a state costs (written, packed, read: 1 us per head at
// d = 64, order 2) does not.
int long_window(const fastmax_problem* pb) {
  return pb->order == 1 ? 512 : pb->d == 64 ? 1536 : 768;
}
struct LongGeo {
  int L, ns;         // window, states per head (segments before the last, or after the first)
  int rows;          // state rows
  size_t raw, packed, cst;
};
LongGeo long_geo(const fastmax_problem* pb) {
  LongGeo g;
  const size_t bh = (size_t)pb->batch * pb->heads;
  const int nb = pb->d / 8, npair = nb * (nb + 1) / 2;
  g.L = pb->causal ? long_window(pb) : 0;
  g.ns = pb->causal ? (pb->nk + g.L - 1) / g.L - 1 : 1;
  g.rows = (pb->order == 2 ? 64 * npair : 0) + pb->d + 1;
  g.raw = up256(bh * (g.ns + 1) * g.rows * (pb->d + 4) * sizeof(float));   // (+ 1: a prompt's last segment)
  g.packed = up256(bh * g.ns * (npair + 1) * (size_t)(pb->d / 8 + 2) * 1024);
  g.cst = up256(bh * g.ns * (pb->d + 8) * sizeof(float));
  return g;
}
fastmax_tensor after(const fastmax_tensor& t, int tokens, int es) {
  fastmax_tensor r = t;
  r.ptr = (char*)t.ptr + (int64_t)tokens * t.stride_n * es;
  return r;
}
bool f32_map(CUtensorMap* m, float* p, const fastmax_problem* pb, int n, int rows) {
  const int64_t bh = (int64_t)pb->batch * pb->heads;
  return tc_make_map(m, fastmax_tensor{p, bh * n * pb->d, (int64_t)n * pb->d, pb->d}, 1, (int)bh, n, 32, rows, true, pb->d, true);
}
void launch_pack(const fastmax_problem* pb, const LongGeo& g, const float* raw, uint8_t* S, float* cst, bool reverse, float* total, cudaStream_t st) {
  const float c0 = pb->a0, c1 = pb->a1 * pb->inv_temperature, c2 = pb->order == 2 ? pb->a2 * pb->inv_temperature * pb->inv_temperature : 0.f;
  const int nb = pb->d / 8, units = (pb->order == 2 ? nb * (nb + 1) / 2 : 0) + 1;
  const dim3 grid((unsigned)units, (unsigned)(pb->batch * pb->heads));
  LaunchScope ls(KK_WINDOW_PACK, st);
  if (pb->d == 64) lng::pack_kernel<64><<<grid, 640, 0, st>>>(raw, S, cst, g.ns, reverse, pb->order, c0, c1, c2, total);
  else lng::pack_kernel<32><<<grid, 384, 0, st>>>(raw, S, cst, g.ns, reverse, pb->order, c0, c1, c2, total);
}
int sm_total() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}
template <typename K, typename MAPS, typename PARAMS>
cudaError_t launch_items(K kernel, std::atomic<bool>* done, int bytes, int threads, const MAPS& M, const PARAMS& P, int kind, cudaStream_t st) {
  if (P.nitems <= 0) return cudaSuccess;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
  }
  const int sms = sm_total();
  LaunchScope ls(kind, st);
  kernel<<<dim3((unsigned)(P.nitems < sms ? P.nitems : sms)), threads, bytes, st>>>(M, P);
  return cudaGetLastError();
}
template <int D, bool FWD>
cudaError_t launch_apply(const lng::Maps& M, const lng::Params& P, int kind, cudaStream_t st) {
  static std::atomic<bool> done[64];
  return launch_items(lng::ap::apply_kernel<D, FWD>, done, lng::ap::Lay<D>::BYTES, lng::ap::THREADS, M, P, kind, st);
}
template <int D, bool DK>
cudaError_t launch_chain(const lng::Maps& M, const lng::Params& P, int kind, cudaStream_t st) {
  static std::atomic<bool> done[64];
  return launch_items(lng::ch::chain_kernel<D, DK>, done, lng::ch::Lay<D>::BYTES, lng::ch::THREADS, M, P, kind, st);
}
// tokens [row0, end) of n, state of token r: (r - row0) / L
lng::Params long_params(const fastmax_problem* pb, const LongGeo& g, const uint8_t* S, int n, int row0, int end) {
  lng::Params P{};
  const int nb = pb->d / 8;
  P.S = S;
  P.cst = (const float*)(S + g.packed);
  P.heads = pb->heads;
  P.n = end;
  P.row0 = row0;
  P.seg = g.L > 0 ? g.L : (n + lng::ROWS) / lng::ROWS * lng::ROWS;
  P.ns = g.ns;
  P.items_per_head = (end - row0 + lng::ROWS - 1) / lng::ROWS;
  P.nitems = P.items_per_head * pb->batch * pb->heads;
  P.u0 = pb->order == 2 ? 0 : nb * (nb + 1) / 2;
  P.part = pb->causal ? 1 : 0;
  P.w1 = 1.f;
  return P;
}

}  // namespace

static size_t long_forward_workspace(const fastmax_problem* pb) {
  const LongGeo g = long_geo(pb);
  return g.raw + g.packed + g.cst + up256(tc_moments_scratch(pb, pb->nk)) +
         (pb->causal ? up256((size_t)pb->batch * pb->heads * pb->nq * pb->d * sizeof(float)) : 0);
}
static size_t long_backward_workspace(const fastmax_problem* pb) {
  const LongGeo g = long_geo(pb);
  const size_t bh = (size_t)pb->batch * pb->heads;
  const int n = pb->nq > pb->nk ? pb->nq : pb->nk;
  return g.raw + 2 * (g.packed + g.cst) + up256(tc_moments_scratch(pb, n)) + up256(bh * pb->nq * (pb->d + 16) * 2) +
         up256(bh * nd_ld(pb->nq) * sizeof(float)) + (pb->causal ? 3 * up256(bh * pb->nq * pb->d * sizeof(float)) : 0);
}
// Packed states of the keys before every segment but the first (no mask: of all keys): S, then the constant rows behind it
static cudaError_t long_key_states(const fastmax_problem* pb, const LongGeo& g, const fastmax_tensor& k, const fastmax_tensor& v, float* raw, void* xt,
                                   uint8_t* S, float* total, cudaStream_t st) {
  const cudaError_t e = tc_moments(pb, k, v, pb->causal && !total ? g.ns * g.L : pb->nk, false, g.L, nullptr, raw, xt, st);
  if (e != cudaSuccess) return e;
  launch_pack(pb, g, raw, S, (float*)(S + g.packed), false, total, st);
  return cudaGetLastError();
}

static int long_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, cudaStream_t st) {
  const LongGeo g = long_geo(pb);
  const int bh = pb->batch * pb->heads;
  char* base = (char*)ws;
  float* raw = (float*)base; base += g.raw;
  uint8_t* S = a->key_moments_in ? (uint8_t*)const_cast<float*>(a->key_moments_in) : a->key_moments_out ? (uint8_t*)a->key_moments_out : (uint8_t*)base;
  base += g.packed + g.cst;
  void* xt = base; base += up256(tc_moments_scratch(pb, pb->nk));
  float* part = (float*)base;
  pair::Maps M;
  lng::Maps A;
  if (!tc_make_map(&M.a, a->q, pb->batch, pb->heads, pb->nq, 64, pair::R, true, pb->d) ||
      !tc_make_map(&M.x, a->k, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d) ||
      !tc_make_map(&M.y, a->v, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d) || !out_map(&M.o0, a->o, pb, pb->nq))
    return FASTMAX_ERR_UNSUPPORTED;
  M.b = M.o1 = M.p0 = M.p1 = M.a;
  A.x = A.y = A.part = M.a;
  A.out = M.o0;
  cudaError_t e = cudaSuccess;
  if (pb->causal) {
    if (!f32_map(&M.p0, part, pb, pb->nq, 32) || !f32_map(&A.part, part, pb, pb->nq, 128)) return FASTMAX_ERR_UNSUPPORTED;
    pair::Params P{};
    const bool sq = fill(pb, P);
    P.window = g.L;
    P.part_lo = g.L;
    P.part_hi = 1 << 30;
    P.out0 = view_of(a->o);
    P.out1 = view_of(a->g);
    P.nr = P.nx = pb->nq;
    P.ntiles = tiles(pb->nq, 2 * pair::R);
    P.vec0 = 1;
    if (sq) P.w1 = P.c2;
    LaunchScope ls(KK_PAIR_FWD, st);
    e = sq ? launch_d<pair::FWD, true>(pb->d, M, P, bh, st) : launch_d<pair::FWD, false>(pb->d, M, P, bh, st);
  }
  if (e == cudaSuccess && (!a->key_moments_in || a->state_out)) e = long_key_states(pb, g, a->k, a->v, raw, xt, S, a->state_out, st);
  lng::Params P = long_params(pb, g, S, pb->nq, g.L, pb->nq);
  P.g = view_of(a->g);
  if (e == cudaSuccess) e = pb->d == 64 ? launch_apply<64, true>(A, P, KK_WINDOW_FWD, st) : launch_apply<32, true>(A, P, KK_WINDOW_FWD, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

static int long_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, cudaStream_t st) {
  const LongGeo g = long_geo(pb);
  const int bh = pb->batch * pb->heads, d = pb->d, ld = d + 16;
  char* base = (char*)ws;
  float* raw = (float*)base; base += g.raw;
  uint8_t* S = a->key_moments_in ? (uint8_t*)const_cast<float*>(a->key_moments_in) : (uint8_t*)base; base += g.packed + g.cst;
  uint8_t* dS = (uint8_t*)base; base += g.packed + g.cst;
  void* xt = base; base += up256(tc_moments_scratch(pb, pb->nq > pb->nk ? pb->nq : pb->nk));
  __nv_bfloat16* dop = (__nv_bfloat16*)base; base += up256((size_t)bh * pb->nq * ld * 2);
  float* nd = (float*)base; base += up256((size_t)bh * nd_ld(pb->nq) * sizeof(float));
  const size_t pbytes = up256((size_t)bh * pb->nq * d * sizeof(float));
  float *pq = (float*)base, *pk = (float*)(base + pbytes), *pv = (float*)(base + 2 * pbytes);
  const fastmax_tensor dflat{dop, (int64_t)bh * pb->nq * ld, (int64_t)pb->nq * ld, ld};                   // one batch of bh heads
  const fastmax_tensor dhead{dop, (int64_t)pb->heads * pb->nq * ld, (int64_t)pb->nq * ld, ld};
  pair::Maps M, N;   // M: dq, N: dk and dv
  if (!tc_make_map(&M.x, a->k, pb->batch, pb->heads, pb->nk, 64, pair::T, true, d) ||
      !tc_make_map(&M.y, a->v, pb->batch, pb->heads, pb->nk, 64, pair::T, true, d) ||
      !tc_make_map(&M.a, a->q, pb->batch, pb->heads, pb->nq, 64, pair::R, true, d) ||
      !tc_make_map(&M.b, dflat, 1, bh, pb->nq, 64, pair::R, true, d) || !out_map(&M.o0, a->dq, pb, pb->nq) || !out_map(&N.o0, a->dk, pb, pb->nk) ||
      !out_map(&N.o1, a->dv, pb, pb->nk))
    return FASTMAX_ERR_UNSUPPORTED;
  N.x = M.a; N.y = M.b; N.a = M.x; N.b = M.y;
  M.o1 = M.o0;
  M.p0 = M.p1 = N.p0 = N.p1 = M.a;
  lng::Maps Q, K, V;   // dq, dk, dv
  Q.x = M.a; Q.y = M.b; Q.out = M.o0; Q.part = M.a;
  K.x = M.x; K.y = M.y; K.out = N.o0; K.part = M.a;
  V.x = M.x; V.y = M.x; V.out = N.o1; V.part = M.a;
  if (pb->causal && (!f32_map(&M.p0, pq, pb, pb->nq, 32) || !f32_map(&N.p0, pk, pb, pb->nk, 32) || !f32_map(&N.p1, pv, pb, pb->nk, 32) ||
                     !f32_map(&Q.part, pq, pb, pb->nq, 128) || !f32_map(&K.part, pk, pb, pb->nk, 128) || !f32_map(&V.part, pv, pb, pb->nk, 128)))
    return FASTMAX_ERR_UNSUPPORTED;
  cudaError_t e = launch_prologue_any(pb, a, dop, nd, ld, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  if (pb->causal) {
    pair::Params P{};
    const bool sq = fill(pb, P);
    P.window = g.L;
    P.ndelta = nd;
    P.nd_ld = nd_ld(pb->nq);
    P.nr = P.nx = pb->nq;
    P.ntiles = tiles(pb->nq);
    P.vec0 = P.vec1 = 1;
    pair::Params B = P;
    B.part_lo = 0;
    B.part_hi = g.ns * g.L;   // the last window's keys have no later queries
    B.out0 = view_of(a->dk);
    B.out1 = view_of(a->dv);
    if (sq) { B.w0 = 2.f * B.c2; B.w1 = B.c2; P.w0 = 2.f * P.c2; }
    {
      LaunchScope ls(KK_PAIR_BWD_KV, st);
      e = sq ? launch_d<pair::DKV, true>(d, N, B, bh, st) : launch_d<pair::DKV, false>(d, N, B, bh, st);
    }
    P.part_lo = g.L;
    P.part_hi = 1 << 30;
    P.out0 = P.out1 = view_of(a->dq);
    LaunchScope ls(KK_PAIR_BWD_Q, st);
    if (e == cudaSuccess) e = sq ? launch_d<pair::DQ, true>(d, M, P, bh, st) : launch_d<pair::DQ, false>(d, M, P, bh, st);
  }
  if (e == cudaSuccess && !a->key_moments_in) e = long_key_states(pb, g, a->k, a->v, raw, xt, S, nullptr, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  // gradient moments of every segment but the first (no mask: of all queries); raw may be reused: the stream orders it
  e = tc_moments(pb, after(a->q, g.L, 2), after(dhead, g.L, 2), pb->nq - g.L, true, g.L, nullptr, raw, xt, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  launch_pack(pb, g, raw, dS, (float*)(dS + g.packed), true, nullptr, st);
  e = cudaGetLastError();
  lng::Params P = long_params(pb, g, S, pb->nq, g.L, pb->nq);
  P.ndelta = nd;
  P.nd_ld = nd_ld(pb->nq);
  if (e == cudaSuccess) e = d == 64 ? launch_chain<64, false>(Q, P, KK_WINDOW_BWD_Q, st) : launch_chain<32, false>(Q, P, KK_WINDOW_BWD_Q, st);
  P = long_params(pb, g, dS, pb->nk, 0, pb->causal ? g.ns * g.L : pb->nk);
  if (e == cudaSuccess) e = d == 64 ? launch_chain<64, true>(K, P, KK_WINDOW_BWD_K, st) : launch_chain<32, true>(K, P, KK_WINDOW_BWD_K, st);
  if (e == cudaSuccess) e = d == 64 ? launch_apply<64, false>(V, P, KK_WINDOW_BWD_V, st) : launch_apply<32, false>(V, P, KK_WINDOW_BWD_V, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

// ---- long float32 sequences (long_f32.cuh) --------------------------------------------------------------------------------
namespace {

LongGeo long_geo_f32(const fastmax_problem* pb) {
  LongGeo g;
  const size_t bh = (size_t)pb->batch * pb->heads;
  // window: 8 heads of 131072 tokens forward + backward 4.26 / 4.49 / 4.85 / 5.27 ms for 256 / 512 / 768 / 1024; the states, which a
  // training call keeps, take half the memory at 512 (414 MB there)
  g.L = 512;
  g.ns = (pb->nk + g.L - 1) / g.L - 1;
  g.rows = (pb->order == 2 ? 64 * lng::f32::NPAIR : 0) + pb->d + 1;
  g.raw = up256(bh * g.ns * g.rows * lng::f32::LD * sizeof(float));
  g.packed = up256(bh * g.ns * lng::f32::UNITS * (size_t)lng::f32::UNIT);
  g.cst = up256(bh * g.ns * lng::f32::CST * sizeof(float));
  return g;
}
bool view_map_f32(CUtensorMap* m, const fastmax_tensor& t, const fastmax_problem* pb, int n, int rows, bool swizzle) {
  return tc_make_map(m, t, pb->batch, pb->heads, n, 32, rows, swizzle, pb->d, true);
}
// the three pieces of [dO' | -delta] or [v | 1] as 128-row boxes of 48 columns
bool g_map_f32(CUtensorMap* m, void* p, const fastmax_problem* pb, int n) {
  const int64_t bh = (int64_t)pb->batch * pb->heads, ld = lng::f32::NC;
  return tc_make_map(m, fastmax_tensor{p, bh * n * ld, n * ld, ld}, 3, (int)bh, n, (int)ld, 128, false, (int)ld);
}
// packed states of x (keys or queries) and y (pieces with 48 columns), rows [first, n): S, then the constant rows behind it
cudaError_t long_states_f32(const fastmax_problem* pb, const LongGeo& g, const fastmax_tensor& x, void* y, int n_all, int first, int n, bool reverse, float* raw,
                            uint8_t* S, cudaStream_t st) {
  using namespace lng::f32;
  mo::Maps M;
  if (!view_map_f32(&M.x, after(x, first, 4), pb, n - first, CHUNK, false) || !pieces_map(&M.y, y, pb, n_all, CHUNK, NC, NC, first)) return cudaErrorInvalidValue;
  mo::Params P{};
  P.out = raw;
  P.n = n - first;
  P.heads = pb->heads;
  P.seg = g.L;
  P.nsplit = g.ns;
  P.tile_first = pb->order == 2 ? 0 : mo::LIN;
  P.nslices = pb->order == 2 ? 3 : 1;
  P.nitems = P.nslices * g.ns * pb->batch * pb->heads;
  P.state_rows = g.rows;
  static std::atomic<bool> done[64];
  cudaError_t e = launch_items(mo::moments_kernel, done, mo::BYTES, mo::THREADS, M, P, KK_TC_MOMENTS, st);
  if (e != cudaSuccess) return e;
  const float c0 = pb->a0, c1 = pb->a1 * pb->inv_temperature, c2 = pb->order == 2 ? pb->a2 * pb->inv_temperature * pb->inv_temperature : 0.f;
  const dim3 grid((unsigned)((pb->order == 2 ? UNITS : 1) + 1), NC / 8, (unsigned)(pb->batch * pb->heads));
  LaunchScope ls(KK_WINDOW_PACK, st);
  pack_kernel<<<grid, 64, 0, st>>>(raw, S, (float*)(S + g.packed), g.ns, reverse, pb->order, c0, c1, c2);
  return cudaGetLastError();
}
template <bool FWD>
cudaError_t launch_apply_f32(const lng::Maps& M, const lng::Params& P, int kind, cudaStream_t st) {
  static std::atomic<bool> done[64];
  return launch_items(lng::f32::ap::apply_kernel<FWD>, done, lng::f32::ap::BYTES, lng::f32::ap::THREADS, M, P, kind, st);
}
cudaError_t launch_chain_f32(const lng::Maps& M, const lng::Params& P, int kind, cudaStream_t st) {
  static std::atomic<bool> done[64];
  return launch_items(lng::f32::ch::chain_kernel, done, lng::f32::ch::BYTES, lng::f32::ch::THREADS, M, P, kind, st);
}

}  // namespace

static size_t long_f32_forward_workspace(const fastmax_problem* pb) {
  const LongGeo g = long_geo_f32(pb);
  return g.raw + g.packed + g.cst + pieces_bytes(pb, pb->nq) + pieces_bytes(pb, pb->nk) + pieces_bytes(pb, pb->nk, lng::f32::NC);
}
static size_t long_f32_backward_workspace(const fastmax_problem* pb) {
  const LongGeo g = long_geo_f32(pb);
  return g.raw + 2 * (g.packed + g.cst) + 2 * pieces_bytes(pb, pb->nq) + 2 * pieces_bytes(pb, pb->nk, lng::f32::NC) +
         up256((size_t)pb->batch * pb->heads * nd_ld(pb->nq) * sizeof(float));
}

static int long_f32_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, cudaStream_t st) {
  const LongGeo g = long_geo_f32(pb);
  const int bh = pb->batch * pb->heads, n = pb->nq;
  char* base = (char*)ws;
  float* raw = (float*)base; base += g.raw;
  uint8_t* S = a->key_moments_in ? (uint8_t*)const_cast<float*>(a->key_moments_in) : a->key_moments_out ? (uint8_t*)a->key_moments_out : (uint8_t*)base;
  base += g.packed + g.cst;
  void *qp = base, *kp = base + pieces_bytes(pb, n), *vp = base + 2 * pieces_bytes(pb, n);
  pair::Maps M;
  lng::Maps A;
  if (!pieces_map(&M.a, qp, pb, n, pair::R) || !pieces_map(&M.x, kp, pb, n, pair::f32::TF) || !pieces_map(&M.y, vp, pb, n, pair::f32::TF, lng::f32::NC) ||
      !view_map_f32(&A.x, a->q, pb, n, 128, true) || !view_map_f32(&A.part, a->o, pb, n, 128, true) || !view_map_f32(&A.out, a->o, pb, n, 32, true))
    return FASTMAX_ERR_UNSUPPORTED;
  M.b = M.o0 = M.o1 = M.p0 = M.p1 = M.a;
  A.y = A.x;
  cudaError_t e = launch_split(pb, pair::f32::SplitArgs{{view_of(a->q), view_of(a->k), view_of(a->v)},
                                                        {(__nv_bfloat16*)qp, (__nv_bfloat16*)kp, (__nv_bfloat16*)vp}, {n, n, n}, {pb->d, pb->d, lng::f32::NC}}, 3, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  {
    pair::Params P{};
    fill(pb, P);
    P.window = P.part_lo = g.L;
    P.part_hi = 1 << 30;
    P.out0 = view_of(a->o);
    P.out1 = view_of(a->g);
    P.nr = P.nx = n;
    P.ntiles = tiles(n);
    P.vec0 = 1;   // (see forward_form)
    LaunchScope ls(KK_PAIR_F32_FWD, st);
    e = launch_f32_d<pair::FWD>(pb, M, P, st);
  }
  if (e == cudaSuccess && !a->key_moments_in) e = long_states_f32(pb, g, a->k, vp, n, 0, g.ns * g.L, false, raw, S, st);
  lng::Params P = long_params(pb, g, S, n, g.L, n);
  P.g = view_of(a->g);
  if (e == cudaSuccess) e = launch_apply_f32<true>(A, P, KK_WINDOW_FWD, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

static int long_f32_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, cudaStream_t st) {
  using lng::f32::NC;
  const LongGeo g = long_geo_f32(pb);
  const int bh = pb->batch * pb->heads, n = pb->nq;
  const size_t narrow = pieces_bytes(pb, n), wide = pieces_bytes(pb, n, NC);
  char* base = (char*)ws;
  float* raw = (float*)base; base += g.raw;
  uint8_t* S = a->key_moments_in ? (uint8_t*)const_cast<float*>(a->key_moments_in) : (uint8_t*)base; base += g.packed + g.cst;
  uint8_t* dS = (uint8_t*)base; base += g.packed + g.cst;
  void *qp = base, *kp = base + narrow, *vp = base + 2 * narrow, *dp = base + 2 * narrow + wide;
  float* nd = (float*)(base + 2 * narrow + 2 * wide);
  pair::Maps M, N;   // M: dq, N: dk and dv
  lng::Maps Q, K, V;
  if (!pieces_map(&M.a, qp, pb, n, pair::R) || !pieces_map(&M.b, dp, pb, n, pair::R, NC) || !pieces_map(&M.x, kp, pb, n, pair::f32::TF) ||
      !pieces_map(&M.y, vp, pb, n, pair::f32::TF, NC) || !pieces_map(&N.a, kp, pb, n, pair::R) || !pieces_map(&N.b, vp, pb, n, pair::R, NC) ||
      !pieces_map(&N.x, qp, pb, n, pair::f32::TF) || !pieces_map(&N.y, dp, pb, n, pair::f32::TF, NC) ||
      !view_map_f32(&Q.x, a->q, pb, n, 128, true) || !view_map_f32(&K.x, a->k, pb, n, 128, true) ||
      !view_map_f32(&Q.part, a->dq, pb, n, 128, true) || !view_map_f32(&Q.out, a->dq, pb, n, 32, true) ||
      !view_map_f32(&K.part, a->dk, pb, n, 128, true) || !view_map_f32(&K.out, a->dk, pb, n, 32, true) ||
      !view_map_f32(&V.part, a->dv, pb, n, 128, true) || !view_map_f32(&V.out, a->dv, pb, n, 32, true) ||
      !g_map_f32(&Q.y, dp, pb, n) || !g_map_f32(&K.y, vp, pb, n))
    return FASTMAX_ERR_UNSUPPORTED;
  M.o0 = M.o1 = M.p0 = M.p1 = N.o0 = N.o1 = N.p0 = N.p1 = M.a;
  V.x = K.x;
  V.y = K.y;
  cudaError_t e = launch_split(pb, pair::f32::SplitArgs{{view_of(a->q), view_of(a->k), view_of(a->v)},
                                                        {(__nv_bfloat16*)qp, (__nv_bfloat16*)kp, (__nv_bfloat16*)vp}, {n, n, n}, {pb->d, pb->d, NC}}, 3, st);
  if (e == cudaSuccess) {
    LaunchScope ls(KK_PROLOGUE, st);
    e = launch_prologue_f32<float, 32>(pb, a, (__nv_bfloat16*)dp, nd, NC, st);
  }
  if (e != cudaSuccess) return report_cuda_error(e);
  pair::Params P{};
  fill(pb, P);
  P.window = g.L;
  P.ndelta = nd;
  P.nd_ld = nd_ld(n);
  P.nr = P.nx = n;
  P.ntiles = tiles(n);
  P.vec0 = P.vec1 = 1;   // (see backward_form)
  pair::Params B = P;
  B.out0 = view_of(a->dk);
  B.out1 = view_of(a->dv);
  {
    LaunchScope ls(KK_PAIR_F32_BWD_KV, st);
    e = launch_f32_d<pair::DKV>(pb, N, B, st);
  }
  P.out0 = P.out1 = view_of(a->dq);
  if (e == cudaSuccess) {
    LaunchScope ls(KK_PAIR_F32_BWD_Q, st);
    e = launch_f32_d<pair::DQ>(pb, M, P, st);
  }
  if (e == cudaSuccess && !a->key_moments_in) e = long_states_f32(pb, g, a->k, vp, n, 0, g.ns * g.L, false, raw, S, st);
  // gradient moments of every segment but the first; raw may be reused: the stream orders it
  if (e == cudaSuccess) e = long_states_f32(pb, g, a->q, dp, n, g.L, n, true, raw, dS, st);
  if (e == cudaSuccess) e = launch_chain_f32(Q, long_params(pb, g, S, n, g.L, n), KK_WINDOW_BWD_Q, st);
  const lng::Params R = long_params(pb, g, dS, n, 0, g.ns * g.L);
  if (e == cudaSuccess) e = launch_chain_f32(K, R, KK_WINDOW_BWD_K, st);
  if (e == cudaSuccess) e = launch_apply_f32<false>(V, R, KK_WINDOW_BWD_V, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

bool pair_packs_key_moments(const fastmax_problem* pb, const fastmax_forward_args* a) {
  fastmax_forward_args train = *a;
  train.state_out = nullptr;
  train.key_moments_in = nullptr;
  train.key_moments_out = (float*)a->q.ptr;
  return forward_form(pb, &train) == 2;
}
// one float more than the states take: every array of segment sums is a multiple of 16 bytes, so a size tells the form
size_t pair_key_moments_bytes(const fastmax_problem* pb) {
  const LongGeo g = pb->dtype == FASTMAX_F32 ? long_geo_f32(pb) : long_geo(pb);
  return g.packed + g.cst + sizeof(float);
}
bool pair_reads_key_moments(const fastmax_problem* pb, const fastmax_backward_args* a) { return backward_form(pb, a) == 2; }

int pair_forward(const fastmax_problem* pb, const fastmax_forward_args* a, void* ws, cudaStream_t st) {
  if (forward_form(pb, a) == 2) return pb->dtype == FASTMAX_F32 ? long_f32_forward(pb, a, ws, st) : long_forward(pb, a, ws, st);
  if (float32_weights(pb)) return pair_f32_forward(pb, a, ws, st);
  pair::Maps M;
  if (!tc_make_map(&M.a, a->q, pb->batch, pb->heads, pb->nq, 64, pair::R, true, pb->d) ||
      !tc_make_map(&M.x, a->k, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d) ||
      !tc_make_map(&M.y, a->v, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d))
    return FASTMAX_ERR_UNSUPPORTED;
  M.b = M.o0 = M.o1 = M.a;
  pair::Params P{};
  const bool sq = fill(pb, P);
  P.out0 = view_of(a->o);
  P.out1 = view_of(a->g);
  P.nr = pb->nq;
  P.nx = pb->nk;
  P.ntiles = tiles(pb->nq, 2 * pair::R);
  P.vec0 = out_map(&M.o0, a->o, pb, pb->nq);
  if (sq) P.w1 = P.c2;
  const int bh = pb->batch * pb->heads;
  LaunchScope ls(KK_PAIR_FWD, st);
  const cudaError_t e = sq ? launch_d<pair::FWD, true>(pb->d, M, P, bh, st) : launch_d<pair::FWD, false>(pb->d, M, P, bh, st);
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

int pair_backward(const fastmax_problem* pb, const fastmax_backward_args* a, void* ws, cudaStream_t st) {
  if (backward_form(pb, a) == 2) return pb->dtype == FASTMAX_F32 ? long_f32_backward(pb, a, ws, st) : long_backward(pb, a, ws, st);
  if (float32_weights(pb)) return pair_f32_backward(pb, a, ws, st);
  const int bh = pb->batch * pb->heads;
  __nv_bfloat16* dop = (__nv_bfloat16*)ws;
  float* nd = (float*)((char*)ws + up256((size_t)bh * pb->nq * pb->d * 2));
  const fastmax_tensor dopt{dop, (int64_t)bh * pb->nq * pb->d, (int64_t)pb->nq * pb->d, pb->d};   // one batch of bh heads
  pair::Maps M;   // dq: held q, dO', streamed k, v
  if (!tc_make_map(&M.x, a->k, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d) ||
      !tc_make_map(&M.y, a->v, pb->batch, pb->heads, pb->nk, 64, pair::T, true, pb->d) ||
      !tc_make_map(&M.a, a->q, pb->batch, pb->heads, pb->nq, 64, pair::R, true, pb->d) ||
      !tc_make_map(&M.b, dopt, 1, bh, pb->nq, 64, pair::R, true, pb->d))
    return FASTMAX_ERR_UNSUPPORTED;
  M.o0 = M.o1 = M.a;
  pair::Maps N;   // dk, dv: the other way round (held and streamed tiles have the same 128-row box)
  N.x = M.a; N.y = M.b; N.a = M.x; N.b = M.y; N.o0 = N.o1 = M.a;
  cudaError_t e = launch_prologue_any(pb, a, dop, nd, pb->d, st);
  if (e != cudaSuccess) return report_cuda_error(e);
  pair::Params P{};
  const bool sq = fill(pb, P);
  P.ndelta = nd;
  P.nd_ld = nd_ld(pb->nq);
  pair::Params K = P;
  K.out0 = view_of(a->dk);
  K.out1 = view_of(a->dv);
  K.nr = pb->nk;
  K.nx = pb->nq;
  K.ntiles = tiles(pb->nk);
  K.vec0 = out_map(&N.o0, a->dk, pb, pb->nk);
  K.vec1 = out_map(&N.o1, a->dv, pb, pb->nk);
  if (sq) { K.w0 = 2.f * K.c2; K.w1 = K.c2; }
  {
    LaunchScope ls(KK_PAIR_BWD_KV, st);
    e = sq ? launch_d<pair::DKV, true>(pb->d, N, K, bh, st) : launch_d<pair::DKV, false>(pb->d, N, K, bh, st);
  }
  if (e != cudaSuccess) return report_cuda_error(e);
  P.out0 = P.out1 = view_of(a->dq);
  P.nr = pb->nq;
  P.nx = pb->nk;
  P.ntiles = tiles(pb->nq);
  P.vec0 = out_map(&M.o0, a->dq, pb, pb->nq);
  if (sq) P.w0 = 2.f * P.c2;
  {
    LaunchScope ls(KK_PAIR_BWD_Q, st);
    e = sq ? launch_d<pair::DQ, true>(pb->d, M, P, bh, st) : launch_d<pair::DQ, false>(pb->d, M, P, bh, st);
  }
  return e == cudaSuccess ? FASTMAX_OK : report_cuda_error(e);
}

int pair_status(int* out) {
  cudaError_t e = cudaMemcpyFromSymbol(out, pair::g_status, sizeof(int), 0, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return report_cuda_error(e);
  if (*out != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(pair::g_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice);
  }
  return FASTMAX_OK;
}
int pair_wait_histogram(int* out, int n) {   // adds to out
  int h[256];
  cudaError_t e = cudaMemcpyFromSymbol(h, pair::g_wait_hist, sizeof(h), 0, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return report_cuda_error(e);
  for (int i = 0; i < n && i < 256; ++i) out[i] += h[i];
  static const int zeros[256] = {0};
  cudaMemcpyToSymbol(pair::g_wait_hist, zeros, sizeof(zeros), 0, cudaMemcpyHostToDevice);
  return FASTMAX_OK;
}

}  // namespace fm
