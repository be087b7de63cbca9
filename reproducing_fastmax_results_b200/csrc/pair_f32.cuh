// Pairwise kernels with float32 weights: float32 tensors, and bf16 heads of 16 dims.  Included by pair_kernels.cu inside fm::pair.
//
// Every float32 operand is the exact sum of three bf16 numbers (8 + 8 + 8 bits), so a product is the sum of the six piece
// products that reach 2^-24 of the largest: hi hi, hi mid, mid hi, mid mid, hi lo, lo hi.  q, k, v and dO' are split once, by
// a pass over memory; P and dS are split in registers.  Six bf16 products run at 1/6 of the bf16 rate, still four times the
// FFMA pipe's.
//
// The tensor pipe adds into its float32 accumulator with truncation: 1e-7 of the value per addition when the terms have one
// sign (measured: 3e-7 after 16 additions, 8e-5 after 1024).  So a chain is kept short: the second products start from zero
// for every streamed tile (64 rows: four additions of hi hi behind the twenty small ones, which go first) and the
// element-wise warps add the tile's result to float32 totals in registers, rounding to nearest.
//
// Measured: 128 heads of 1024 x 64, causal, forward + backward with splitting 13400 us in the CUDA-core engine (FFMA), 520 here
// (each launch by itself: forward 110, dq 135, dk / dv 185, splitting 78 in two passes, dO' 25; back to back they overlap); bf16, 128 heads of 1024 x 16 (q, k, v are one piece each: 1 or 3
// products instead of 6, no pass that splits) 771 and 216.  Bound by the chain scores -> element-wise -> second products
// between few warps (tensor pipe active in 51 to 65 % of the clocks at 64 dims, issue slots 30 %).  What took the forward from 131
// to 110, dq from 156 to 135 and dk / dv from 216 to 185: scores in two blocks (product2), the results of a tile added up behind
// the next tile's P instead of before it (dq: before its arithmetic, when its products have ended), rows written 16 bytes a
// thread (one row per instruction, the warps that write dk and dv held up the next item for 7000 clocks), and the forward's held
// tile of the next item loaded early.
//
// Roles and hand-offs are those of the bf16 kernels; the streamed pair's two tiles have barriers of their own, because with
// three pieces each only two or three stages fit and each tile can be let go at a different time.
#pragma once

namespace f32 {

constexpr int EW = 8, ROLES = EW + 3, THREADS = (W_EW + EW) * 32;   // element-wise warps: TMEM lane quarters x 32-column halves
constexpr int TF = 64;                       // streamed rows per tile
constexpr int XF = TF * 128;                 // one piece of a streamed tile
constexpr int AF = R * 128;                  // one piece of a held tile
template <int KIND>
struct Lay {
  static constexpr int SETS = KIND == FWD ? 2 : 1;                    // held sets
  static constexpr int HELD = (KIND == FWD ? 3 : 6) * AF;
  static constexpr int STAGES = 2;
  static constexpr int STAGE = 6 * XF;       // X pieces, then Y pieces
  static constexpr int OFF_X = SETS * HELD;
  static constexpr int OFF_OUT = OFF_X + STAGES * STAGE;   // 4 KB of output staging per warp that writes rows
  static constexpr int OFF_ND = OFF_OUT + (KIND == DKV ? 4 : EW) * 4096;   // DKV: -delta of the streamed queries per stage
  static constexpr int OFF_CLC = OFF_ND + STAGES * TF * 4;
  static constexpr int OFF_BAR = OFF_CLC + 16 * CLC;
  static constexpr int BYTES = OFF_BAR + 512 + 1024;
};
static_assert(Lay<FWD>::BYTES <= 232448 && Lay<DQ>::BYTES <= 232448 && Lay<DKV>::BYTES <= 232448, "shared memory budget");
constexpr int B_FX = 0, B_FY = 2, B_EX = 4, B_EY = 6, B_HFULL = 8, B_HEMPTY = 10, B_S = 12, B_READ = 14, B_P = 15, B_ACC = 17, B_AFREE = 19,
              B_CFULL = 21, B_CEMPTY = B_CFULL + CLC, B_DRAIN = B_CEMPTY + CLC, B_COUNT = B_DRAIN + 2;
// TMEM columns.  S (and DQ: dP) in two blocks of 64 columns, the small piece products in the second; P and dS in three pieces of
// 32 columns.  What a tile leaves (P or dS, its results) is doubled where there is room, so that the element-wise warps go on
// with the next tile while its second products run.
template <int KIND>
struct Cols {
  static constexpr uint32_t NACC = KIND == FWD ? 2 : 1, NP = KIND == DKV ? 1 : 2;   // results, P / dS
  static constexpr uint32_t ACC = 0, ACC1 = 64, S = KIND == DQ ? 64 : 128, DP = KIND == DQ ? 192 : 256;   // DKV: dv, dk
  static constexpr uint32_t P = KIND == FWD ? 256 : 320, DS = KIND == DKV ? 416 : 320;
  static constexpr uint32_t SUM = 448;   // FWD: row sums of the two halves, of the last four items
};
// dk / dv: a warpgroup of its own adds up the accumulators (128 totals per thread: beside a tile they do not fit into the
// element-wise warps' registers; spilled, the kernel took four times as long).  Registers are moved between the warpgroups.
constexpr int W_SUM = W_EW + EW;
template <int KIND>
constexpr int THREADS_F = KIND == DKV ? (W_SUM + 4) * 32 : THREADS;
constexpr int REG_LAUNCH = 128, REG_REST = 48, REG_EW = 136, REG_SUM = 192;
static_assert(REG_REST * W_EW + REG_EW * EW + REG_SUM * 4 <= REG_LAUNCH * (W_SUM + 4), "setmaxnreg.inc waits for registers the block does not have");

// the piece products that count, the smallest first
__device__ constexpr int PIECE_A[6] = {0, 2, 1, 0, 1, 0}, PIECE_B[6] = {2, 0, 1, 1, 0, 0};

// two float32 numbers -> their three bf16 pieces
__device__ __forceinline__ void split3(uint64_t x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint64_t minus = 0xBF800000BF800000ull;
  hi = bf16x2(x);
  const uint64_t r = fma2(pack2u(hi << 16, hi & 0xffff0000u), minus, x);   // exact
  mid = bf16x2(r);
  lo = bf16x2(fma2(pack2u(mid << 16, mid & 0xffff0000u), minus, r));
}

// waits without an out-of-line call (ptxas cannot allocate a callee under mixed register allowances)
__device__ __forceinline__ void wait_inline(uint64_t* bar, uint32_t parity, int code, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag != 0) return;
    if (clock64() - t0 > WAIT_CYCLES) {
      if (*abort_flag == 0) atomicAdd(&g_wait_hist[code & 255], 1);
      *abort_flag = 1;
      atomicExch(&g_status, code);
      return;
    }
  }
}

// IN: pieces of q, k and v: 3, from a pass over float32 tensors, or 1: bf16 tensors, read as they are (their results are bf16)
template <int D, int KIND, int IN>
__global__ void __launch_bounds__(THREADS_F<KIND>, 1) pair_f32_kernel(const __grid_constant__ Maps M, const Params P) {
  using L = Lay<KIND>;
  constexpr int KS = D / 16, STAGES = L::STAGES;
  constexpr int PY = KIND == DKV ? 3 : IN, PB = KIND == DQ ? 3 : IN;   // dO', wherever it is an operand, has three pieces
  using Out = typename std::conditional<IN == 1, __nv_bfloat16, float>::type;
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
      if (i == B_READ || i == B_P || i == B_P + 1) n = EW;
      if (i == B_AFREE || i == B_AFREE + 1) n = KIND == DKV ? 4 : EW;
      if (i >= B_CEMPTY && i < B_CEMPTY + CLC) n = KIND == DKV ? ROLES + 4 : ROLES;
      mbar_init(&bars[i], n);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (w == W_ACC) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  grid_wait();
  grid_trigger();
  auto WAIT = [&](int bar, uint32_t phase, int code) { wait_inline(&bars[bar], phase & 1u, code, abort_flag); };
  auto next_item = [&](int n) -> int {
    const int c = n & (CLC - 1);
    WAIT(B_CFULL + c, (uint32_t)(n / CLC), 76);
    int idx = *abort_flag != 0 ? -1 : clc_read(sm + L::OFF_CLC + 16 * c);
    fence_proxy_async_smem();
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (lane == 0) mbar_arrive(&bars[B_CEMPTY + c]);
    return idx;
  };
  // DKV: the role branches move registers (inside each branch: past a join of branches ptxas assumes the smaller allowance)
#define FM_REG_DEC() if (KIND == DKV) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REG_REST))
#define FM_REG_INC(n_) if (KIND == DKV) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(n_))
  int issued_x = 0, issued_y = 0, helds = 0, asked = 0;   // what the loader has asked for
  if (w == W_LOAD) {
    FM_REG_DEC();
    // ================= loader and item scheduler =================
    // tile i of the item: the three pieces of one operand
    auto load_tile = [&](const Item& it, int i, bool y) {
      int& issued = y ? issued_y : issued_x;
      const int s = issued % STAGES;
      if (issued >= STAGES) WAIT((y ? B_EY : B_EX) + s, (uint32_t)(issued / STAGES) - 1u, y ? 71 : 70);
      if (*abort_flag != 0) return;
      if (lane == 0) {
        uint8_t* x = sm + L::OFF_X + s * L::STAGE + (y ? 3 * XF : 0);
        uint64_t* bar = &bars[(y ? B_FY : B_FX) + s];
        const int row = (it.t0 + i) * TF;
        const bool nd = KIND == DKV && y;
        const int pieces = y ? PY : IN;
        mbar_arrive_expect_tx(bar, pieces * XF + (nd ? TF * 4 : 0));
        if (pieces == 1) {
          tma_load_4d(x, y ? &M.y : &M.x, bar, 0, row, it.h, it.b);
        } else {
#pragma unroll
          for (int p = 0; p < 3; ++p) tma_load_4d(x + p * XF, y ? &M.y : &M.x, bar, 0, row, it.head, p);
        }
        if (nd) bulk_load(sm + L::OFF_ND + s * TF * 4, P.ndelta + (long long)it.head * P.nd_ld + row, TF * 4, bar);
      }
      ++issued;
    };
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const int c = n & (CLC - 1);
      if (n >= CLC) WAIT(B_CEMPTY + c, (uint32_t)(n / CLC) - 1u, 77);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_CFULL + c], 16);
        clc_try_cancel(sm + L::OFF_CLC + 16 * c, &bars[B_CFULL + c]);
      }
      asked = n + 1;
      const Item it = decode<KIND, TF, R>(idx, P);
      const int hs = n % L::SETS;
      if (n >= L::SETS) WAIT(B_HEMPTY + hs, (uint32_t)(n / L::SETS) - 1u, 78);
      if (*abort_flag != 0) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[B_HFULL + hs], (IN + (KIND == FWD ? 0 : PB)) * AF);
        auto load_held = [&](uint8_t* dst, const CUtensorMap* m, int pieces) {
          if (pieces == 1) tma_load_4d(dst, m, &bars[B_HFULL + hs], 0, it.r0, it.h, it.b);
          else
#pragma unroll
            for (int p = 0; p < 3; ++p) tma_load_4d(dst + p * AF, m, &bars[B_HFULL + hs], 0, it.r0, it.head, p);
        };
        load_held(sm + hs * L::HELD, &M.a, IN);
        if (KIND != FWD) load_held(sm + 3 * AF, &M.b, PB);
      }
      helds = n + 1;
      for (int i = 0; i < it.n0 && *abort_flag == 0; ++i) {   // in the order in which the tiles are used
        load_tile(it, i, KIND == DQ);
        load_tile(it, i, KIND != DQ);
      }
      idx = next_item(n);
    }
  } else if (w == W_SCORE) {
    FM_REG_DEC();
    // ================= issuer of the first products =================
    constexpr uint32_t ID_S = make_idesc_bf16(R, TF, 0, 0), ID_S2 = make_idesc_bf16(R, 2 * TF, 0, 0);
    const uint64_t dH0 = make_smem_desc(smem_u32(sm), 16, 1024, 2);
    const uint64_t dX0 = make_smem_desc(smem_u32(sm + L::OFF_X), 16, 1024, 2);
    // sum over the piece products of a held tile with `na` pieces and a streamed one with `nb`, the smallest first
    auto product = [&](uint32_t acc, uint64_t a, int na, uint64_t b, int nb) {
      bool more = false;
#pragma unroll
      for (int t = 0; t < 6; ++t) {
        if (PIECE_A[t] >= na || PIECE_B[t] >= nb) continue;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          mma_ss_elect(acc, a + (uint64_t)(PIECE_A[t] * (AF >> 4) + 2 * ks), b + (uint64_t)(PIECE_B[t] * (XF >> 4) + 2 * ks), ID_S, more);
          more = true;
        }
      }
    };
    // The same of three pieces each, in two blocks: the streamed tile's hi and mid pieces lie one behind the other and enter as one
    // operand of 128 rows.  A product of 64 columns keeps the pipe for 48 clocks, one of 128 for 64: 896 instead of 1152 a tile.
    auto product2 = [&](uint32_t acc, uint64_t a, uint64_t b) {
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) mma_ss_elect(acc, a + (uint64_t)((AF >> 4) + 2 * ks), b + (uint64_t)(2 * ks), ID_S2, ks > 0);   // mid hi, mid mid
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) mma_ss_elect(acc + 64u, a + (uint64_t)(2 * (AF >> 4) + 2 * ks), b + (uint64_t)(2 * ks), ID_S, 1u);   // lo hi
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) mma_ss_elect(acc + 64u, a + (uint64_t)(2 * ks), b + (uint64_t)(2 * (XF >> 4) + 2 * ks), ID_S, 1u);   // hi lo
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) mma_ss_elect(acc, a + (uint64_t)(2 * ks), b + (uint64_t)(2 * ks), ID_S2, 1u);                      // hi hi, hi mid
    };
    uint32_t k = 0;
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const Item it = decode<KIND, TF, R>(idx, P);
      const int hs = n % L::SETS;
      const uint64_t dH = dH0 + (uint64_t)(hs * (L::HELD >> 4));
      WAIT(B_HFULL + hs, (uint32_t)(n / L::SETS), 72);
      for (int i = 0; i < it.n0; ++i) {
        const uint32_t s = k % STAGES;
        const uint64_t dX = dX0 + (uint64_t)(s * (L::STAGE >> 4)), dY = dX + (uint64_t)(3 * XF >> 4);
        if (k > 0) WAIT(B_READ, k - 1u, 80);   // the last tile's scores and dP have been read
        if (KIND == DQ) {   // v is needed here only: it can go before k, which the second product reads too
          WAIT(B_FY + (int)s, k / STAGES, 74);
          tc_fence_after_sync();
          if constexpr (IN == 3) product2(tmem + Cols<KIND>::DP, dH + (uint64_t)(3 * AF >> 4), dY);
          else product(tmem + Cols<KIND>::DP, dH + (uint64_t)(3 * AF >> 4), PB, dY, PY);
          mma_commit_elect(&bars[B_EY + s]);
        }
        WAIT(B_FX + (int)s, k / STAGES, 73);
        tc_fence_after_sync();
        if constexpr (IN == 3) product2(tmem + Cols<KIND>::S, dH, dX);
        else product(tmem + Cols<KIND>::S, dH, IN, dX, IN);
        if (KIND == FWD) mma_commit_elect(&bars[B_EX + s]);
        if (KIND == DKV) {
          WAIT(B_FY + (int)s, k / STAGES, 74);
          tc_fence_after_sync();
          product(tmem + Cols<KIND>::DP, dH + (uint64_t)(3 * AF >> 4), PB, dY, PY);
        }
        mma_commit_elect(&bars[B_S + (k & 1u)]);
        ++k;
      }
      mma_commit_elect(&bars[B_HEMPTY + hs]);
      idx = next_item(n);
    }
    if (*abort_flag != 0) {
      mma_commit_elect(&bars[B_DRAIN]);
      mbar_wait_bounded(&bars[B_DRAIN], 0, WAIT_CYCLES);
    }
  } else if (w == W_ACC) {
    FM_REG_DEC();
    // ================= issuer of the second products =================
    constexpr uint32_t ID_ACC = make_idesc_bf16(R, D, 0, 1);
    const uint64_t dX0 = make_smem_desc(smem_u32(sm + L::OFF_X), XF, 1024, 2);
    auto product = [&](uint32_t acc, uint32_t a, uint64_t b, int nb) {   // P or dS (three pieces) with a streamed tile
      bool more = false;
#pragma unroll
      for (int t = 0; t < 6; ++t) {
        if (PIECE_B[t] >= nb) continue;
#pragma unroll
        for (int kk = 0; kk < TF / 16; ++kk) {
          mma_ts_elect(acc, a + 32u * PIECE_A[t] + 8u * kk, b + (uint64_t)(PIECE_B[t] * (XF >> 4) + 128 * kk), ID_ACC, more);
          more = true;
        }
      }
    };
    using C = Cols<KIND>;
    uint32_t k = 0;
    int idx = blockIdx.x;
    for (int n = 0; idx >= 0; ++n) {
      const Item it = decode<KIND, TF, R>(idx, P);
      for (int i = 0; i < it.n0; ++i) {
        const uint32_t s = k % STAGES;
        const uint64_t dX = dX0 + (uint64_t)(s * (L::STAGE >> 4)), dY = dX + (uint64_t)(3 * XF >> 4);
        if (KIND == FWD) WAIT(B_FY + (int)s, k / STAGES, 75);
        WAIT(B_P + (int)(k % C::NP), k / C::NP, 79);
        if (k >= C::NACC) WAIT(B_AFREE + (int)(k % C::NACC), k / C::NACC - 1u, 82);   // the results there have been added up
        tc_fence_after_sync();
        if (KIND != FWD) {
          product(tmem + (KIND == DKV ? C::ACC1 : C::ACC), tmem + C::DS + 96u * (k % C::NP), dX, IN);
          mma_commit_elect(&bars[B_EX + s]);
        }
        if (KIND != DQ) {
          product(tmem + C::ACC + 64u * (k % C::NACC), tmem + C::P + 96u * (k % C::NP), dY, PY);
          mma_commit_elect(&bars[B_EY + s]);
        }
        mma_commit_elect(&bars[B_ACC + (int)(k % C::NACC)]);
        ++k;
      }
      idx = next_item(n);
    }
    if (*abort_flag != 0) {
      mma_commit_elect(&bars[B_DRAIN + 1]);
      mbar_wait_bounded(&bars[B_DRAIN + 1], 0, WAIT_CYCLES);
    }
  } else if (w < W_EW) {   // spare
    FM_REG_DEC();
  } else {
    // ================= element-wise warps: TMEM lane quarter x 32-column half of the tile; DKV: + the warps that add up =================
    const int quarter = w & 3, half = (w - W_EW) >> 2;   // half == 2: adding up (DKV)
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    // Totals of this warp: half a row of dq or O'; dv and dk (two rows of D) in the warps that add up
    constexpr int NA = KIND == DKV ? 2 * D : D / 2;
    constexpr uint32_t NACC = Cols<KIND>::NACC, NP = Cols<KIND>::NP;
    constexpr int CH = KIND == DKV ? (D < 32 ? D : 32) : (NA < 32 ? NA : 32);
    auto clear = [&](uint64_t (&tot)[NA / 2]) {
#pragma unroll
      for (int j = 0; j < NA / 2; ++j) tot[j] = 0ull;
    };
    auto drain = [&](uint64_t (&tot)[NA / 2], uint32_t tile) {   // adds the results of a tile's second products
      WAIT(B_ACC + (int)(tile % NACC), tile / NACC, 83);
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < NA / CH; ++c) {
        uint32_t r[CH];
        // DKV: chunks of dv, then of dk
        tmem_ld<CH>(lane_addr + (KIND == DKV ? (uint32_t)(64 * (c * CH / D) + c * CH % D) : 64u * (tile % NACC) + (uint32_t)(half * NA + CH * c)), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < CH / 2; ++j) tot[c * (CH / 2) + j] = add2(tot[c * (CH / 2) + j], pack2u(r[2 * j], r[2 * j + 1]));
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_AFREE + (int)(tile % NACC)]);
    };
    // rows -> shared memory -> whole rows in global memory: 16 bytes a thread where the rows allow it (P.vec0, P.vec1), else element
    // by element (one row per store instruction).  The exchange is free of bank conflicts either way.
    auto write_rows = [&](const Item& it, const uint64_t (&tot)[NA / 2], float wgt) {
      float* stage = reinterpret_cast<float*>(sm + L::OFF_OUT + (KIND == DKV ? quarter : w - W_EW) * 4096);
#pragma unroll
      for (int c = 0; c < NA / CH; ++c) {
        const bool second = KIND == DKV && c * CH < D;
        const View& out = second ? P.out1 : P.out0;
        Out* base = reinterpret_cast<Out*>(const_cast<void*>(out.ptr)) + (long long)it.b * out.sb + (long long)it.h * out.sh +
                    (KIND == DKV ? c * CH % D : half * NA + CH * c);
        __syncwarp();
        if (sizeof(Out) == 4 && CH >= 8 && (second ? P.vec1 : P.vec0)) {
          constexpr int Q = CH / 4;   // 16-byte pieces of a row
#pragma unroll
          for (int j = 0; j < Q; ++j) {
            float4 v;
            unpack2(tot[c * (CH / 2) + 2 * j], v.x, v.y);
            unpack2(tot[c * (CH / 2) + 2 * j + 1], v.z, v.w);
            v.x *= wgt; v.y *= wgt; v.z *= wgt; v.w *= wgt;
            reinterpret_cast<float4*>(stage)[lane * Q + (j ^ (lane & (Q - 1)))] = v;
          }
          __syncwarp();
          const int rr = lane / Q, cc = lane % Q;
#pragma unroll
          for (int r = 0; r < 32; r += 32 / Q) {
            const int g = it.r0 + quarter * 32 + r + rr;
            const float4 v = reinterpret_cast<const float4*>(stage)[(r + rr) * Q + (cc ^ ((r + rr) & (Q - 1)))];
            if (g < P.nr) reinterpret_cast<float4*>(base + (long long)g * out.sn)[cc] = v;
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < CH / 2; ++j) {
          float a, b;
          unpack2(tot[c * (CH / 2) + j], a, b);
          stage[lane * 32 + ((2 * j) ^ lane)] = a * wgt;
          stage[lane * 32 + ((2 * j + 1) ^ lane)] = b * wgt;
        }
        __syncwarp();
        constexpr int RP = 32 / CH;   // rows per instruction
        const int rr = lane / CH, cc = lane % CH;
#pragma unroll 4
        for (int r = 0; r < 32; r += RP) {
          const int g = it.r0 + quarter * 32 + r + rr;
          const float v = stage[(r + rr) * 32 + (cc ^ (r + rr))];
          if (g < P.nr) base[(long long)g * out.sn + cc] = static_cast<Out>(v);
        }
      }
    };
    uint32_t k = 0;
    int idx = blockIdx.x;
    if (KIND == DKV && w >= W_SUM) {
      FM_REG_INC(REG_SUM);
      for (int n = 0; idx >= 0; ++n) {
        const Item it = decode<KIND, TF, R>(idx, P);
        uint64_t tot[NA / 2];
        clear(tot);
        for (int i = 0; i < it.n0; ++i) drain(tot, k++);
        write_rows(it, tot, 1.f);
        idx = next_item(n);
      }
    } else {
      FM_REG_INC(REG_EW);
      const uint64_t C0 = pack2(P.c0, P.c0), C1 = pack2(P.c1, P.c1), C2 = pack2(P.c2, P.c2);
      uint64_t tot[NA / 2];
      bool pend = false;       // the last item's rows are still to be written: they are behind the next item's first tile
      Item last{};
      int last_n = 0;
      auto results = [&] {
        drain(tot, k - 1u);
        float wgt = 1.f;
        if (KIND == FWD) {   // (each half's sum was there before its last P of the item)
          uint32_t h[2];
          tmem_ld2(lane_addr + Cols<KIND>::SUM + 2u * ((uint32_t)last_n & 3u), h);
          tmem_ld_wait();
          const float g = __uint_as_float(h[0]) + __uint_as_float(h[1]);
          wgt = last.r0 >= P.part_lo && last.r0 < P.part_hi ? 1.f : 1.f / g;   // partial rows: not divided yet
          const int row = last.r0 + quarter * 32 + lane;
          if (half == 0 && row < P.nr)
            reinterpret_cast<float*>(const_cast<void*>(P.out1.ptr))[(long long)last.b * P.out1.sb + (long long)last.h * P.out1.sh + (long long)row * P.out1.sn] = g;
        }
        write_rows(last, tot, wgt);
      };
      if (KIND != DKV) clear(tot);
      for (int n = 0; idx >= 0; ++n) {
        const Item it = decode<KIND, TF, R>(idx, P);
        const int row = it.r0 + quarter * 32 + lane;
        uint64_t ND = 0ull;
        if (KIND == DQ) {
          const float nd = row < P.nr ? P.ndelta[(long long)it.head * P.nd_ld + row] : 0.f;
          ND = pack2(nd, nd);
        }
        float total = 0.f;   // FWD: this half's row sum
        for (int i = 0; i < it.n0; ++i) {
          WAIT(B_S + (int)(k & 1u), k >> 1, 84);
          const int s_ = (int)(k % STAGES);
          if (KIND == DKV) WAIT(B_FY + s_, k / STAGES, 81);
          tc_fence_after_sync();
          const int x0 = (it.t0 + i) * TF + half * 32;
          int lo = 0, hi = 32;
          if (KIND == DKV) {
            if (P.causal) lo = row - P.off - x0;
          } else {
            if (P.causal) hi = row + P.off - x0 + 1;
            if (KIND == FWD && P.nx - x0 < hi) hi = P.nx - x0;
          }
          const bool whole = __all_sync(0xffffffffu, lo <= 0 && hi >= 32);
          uint32_t s[32], d[32];
          auto load = [&](uint32_t (&v)[32], uint32_t col, bool both) {   // both blocks of S or dP
            uint32_t small[32];
            tmem_ld32(lane_addr + col + 32u * half, v);
            if (both) tmem_ld32(lane_addr + col + 64u + 32u * half, small);
            if (KIND == DKV) tmem_ld32(lane_addr + Cols<KIND>::DP + 32u * half, d);
            tmem_ld_wait();
            if (both)
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const uint64_t x = add2(pack2u(v[2 * j], v[2 * j + 1]), pack2u(small[2 * j], small[2 * j + 1]));
                v[2 * j] = (uint32_t)x;
                v[2 * j + 1] = (uint32_t)(x >> 32);
              }
          };
          load(s, Cols<KIND>::S, IN == 3);
          if (KIND == DQ) load(d, Cols<KIND>::DP, IN == 3);
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[B_READ]);
          if (KIND == DQ && i > 0) drain(tot, k - 1u);   // (its products ended under the first ones of this tile)
          // values: P in s, dS in d
          const ulonglong2* ndp = reinterpret_cast<const ulonglong2*>(sm + L::OFF_ND + s_ * TF * 4 + half * 128);
          uint64_t sum = 0ull;
#pragma unroll
          for (int j2 = 0; j2 < 8; ++j2) {
            ulonglong2 n2;
            n2.x = n2.y = ND;
            if (KIND == DKV) n2 = ndp[j2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int col = 4 * j2 + 2 * e;
              const bool v0 = whole || (col >= lo && col < hi), v1 = whole || (col + 1 >= lo && col + 1 < hi);
              const uint64_t x = pack2u(s[col], s[col + 1]);
              const uint64_t t = fma2(C2, x, C1);
              if (KIND != DQ) {
                float a, b;
                unpack2(fma2(t, x, C0), a, b);
                if (!whole) { a = v0 ? a : 0.f; b = v1 ? b : 0.f; }
                if (KIND == FWD) sum = add2(sum, pack2(a, b));
                s[col] = __float_as_uint(a);
                s[col + 1] = __float_as_uint(b);
              }
              if (KIND != FWD) {
                float a, b;
                unpack2(mul2(fma2(C2, x, t), add2(pack2u(d[col], d[col + 1]), e ? n2.y : n2.x)), a, b);
                if (!whole) { a = v0 ? a : 0.f; b = v1 ? b : 0.f; }
                d[col] = __float_as_uint(a);
                d[col + 1] = __float_as_uint(b);
              }
            }
          }
          if (KIND == FWD) {
            float a, b;
            unpack2(sum, a, b);
            total += a + b;
            if (i == it.n0 - 1) tmem_st1(lane_addr + Cols<KIND>::SUM + 2u * ((uint32_t)n & 3u) + (uint32_t)half, __float_as_uint(total));
          }
          if (KIND == DKV && k > 0) {   // the last tile's second products are done: P and dS may be overwritten
            WAIT(B_ACC, k - 1u, 85);
            tc_fence_after_sync();
          }
          // in pieces.  (FWD, DQ: the tile before the last one is added up, so these columns are free)
          auto put = [&](const uint32_t (&v)[32], uint32_t addr) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t pp[3][8];
#pragma unroll
              for (int j = 0; j < 8; ++j) split3(pack2u(v[16 * c + 2 * j], v[16 * c + 2 * j + 1]), pp[0][j], pp[1][j], pp[2][j]);
#pragma unroll
              for (int p = 0; p < 3; ++p) tmem_st8(addr + 32u * p + 16u * half + 8u * c, pp[p]);
            }
          };
          if (KIND != DQ) put(s, lane_addr + Cols<KIND>::P + 96u * (k % NP));
          if (KIND != FWD) put(d, lane_addr + Cols<KIND>::DS + 96u * (k % NP));
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars[B_P + (int)(k % NP)]);
          if (KIND != DKV) {
            if (KIND == FWD && i > 0) {
              drain(tot, k - 1u);
            } else if (i == 0 && pend) {
              results();
              clear(tot);
            }
          }
          ++k;
        }
        pend = KIND != DKV;
        last = it;
        last_n = n;
        idx = next_item(n);
      }
      if (pend) results();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0) {
    if (w == W_LOAD) {
      for (int i = issued_x > STAGES ? issued_x - STAGES : 0; i < issued_x; ++i)
        mbar_wait_bounded(&bars[B_FX + i % STAGES], (uint32_t)(i / STAGES) & 1u, WAIT_CYCLES);
      for (int i = issued_y > STAGES ? issued_y - STAGES : 0; i < issued_y; ++i)
        mbar_wait_bounded(&bars[B_FY + i % STAGES], (uint32_t)(i / STAGES) & 1u, WAIT_CYCLES);
      for (int i = helds > L::SETS ? helds - L::SETS : 0; i < helds; ++i)
        mbar_wait_bounded(&bars[B_HFULL + i % L::SETS], (uint32_t)(i / L::SETS) & 1u, WAIT_CYCLES);
      for (int i = asked > CLC ? asked - CLC : 0; i < asked; ++i)
        mbar_wait_bounded(&bars[B_CFULL + (i & (CLC - 1))], (uint32_t)(i / CLC) & 1u, WAIT_CYCLES);
    }
    __syncthreads();
  }
  if (w == W_ACC) tmem_dealloc(tmem, 512);
}

// Splits float32 views into bf16 pieces: out[piece][batch*heads][n][ld], ld = D, or D + 16: [values, 1, 0 ...].  A thread takes
// eight columns; blockIdx.z picks the tensor.
struct SplitArgs {
  View x[3];
  __nv_bfloat16* out[3];
  int n[3], ld[3];
};
__device__ __forceinline__ void store_pieces(__nv_bfloat16* out, long long plane, long long at, const float (&v)[8]) {
  uint32_t r[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) split3(pack2(v[2 * i], v[2 * i + 1]), r[0][i], r[1][i], r[2][i]);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(out + p * plane + at) = make_uint4(r[p][0], r[p][1], r[p][2], r[p][3]);
}
// the sixteen columns behind the values: x, then zeros
__device__ __forceinline__ void store_tail(__nv_bfloat16* out, long long plane, long long at, float x) {
  uint32_t r[3];
  split3(pack2(x, 0.f), r[0], r[1], r[2]);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    uint4* t = reinterpret_cast<uint4*>(out + p * plane + at);
    t[0] = make_uint4(r[p], 0u, 0u, 0u);
    t[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}
template <int D>
__global__ void __launch_bounds__(256) split_kernel(const SplitArgs A, int heads) {
  constexpr int TPR = D / 8;
  grid_wait();
  grid_trigger();
  const int t = blockIdx.z, head = blockIdx.y, b = head / heads, h = head - b * heads;
  const int row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, c = (threadIdx.x % TPR) * 8;
  if (row >= A.n[t]) return;
  const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(A.x[t].ptr) + (long long)b * A.x[t].sb + (long long)h * A.x[t].sh +
                                                    (long long)row * A.x[t].sn + c);
  const float4 u = p[0], w = p[1];
  const float v[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
  const int ld = A.ld[t];
  const long long plane = (long long)gridDim.y * A.n[t] * ld, at = ((long long)head * A.n[t] + row) * ld;
  store_pieces(A.out[t], plane, at + c, v);
  if (c == 0 && ld > D) store_tail(A.out[t], plane, at + D, 1.f);
}

// dO' = dO / g in pieces (ld = D + 16: with -delta behind the values) and -delta = -(dO . o) / g; T: the type of dO and o
template <typename T, int D, bool VEC>
__global__ void __launch_bounds__(256) prologue_f32_kernel(View dout, View o, View g, __nv_bfloat16* __restrict__ dop, float* __restrict__ ndelta,
                                                           int nq, int nd_ld, int heads, int ld) {
  constexpr int TPR = D / 8;
  grid_wait();
  grid_trigger();
  const int head = blockIdx.y, b = head / heads, h = head - b * heads;
  const int row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR, c = (threadIdx.x % TPR) * 8;
  float v[8], dot = 0.f;
  if (row < nq) {
    const T* pd = reinterpret_cast<const T*>(dout.ptr) + (long long)b * dout.sb + (long long)h * dout.sh + (long long)row * dout.sn + c;
    const T* po = reinterpret_cast<const T*>(o.ptr) + (long long)b * o.sb + (long long)h * o.sh + (long long)row * o.sn + c;
    const float inv = 1.f / reinterpret_cast<const float*>(g.ptr)[(long long)b * g.sb + (long long)h * g.sh + (long long)row * g.sn];
    float x[8];
    alignas(16) T td[8], to[8];
    if (VEC) {
#pragma unroll
      for (int i = 0; i < (int)sizeof(T) / 2; ++i) {
        reinterpret_cast<uint4*>(td)[i] = reinterpret_cast<const uint4*>(pd)[i];
        reinterpret_cast<uint4*>(to)[i] = reinterpret_cast<const uint4*>(po)[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) { td[i] = pd[i]; to[i] = po[i]; }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = static_cast<float>(td[i]);
      x[i] = static_cast<float>(to[i]);
      v[i] *= inv;
      dot += v[i] * x[i];
    }
  }
#pragma unroll
  for (int m = TPR / 2; m > 0; m >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, m);
  if (row < nq) {
    const long long plane = (long long)gridDim.y * nq * ld, at = ((long long)head * nq + row) * ld;
    store_pieces(dop, plane, at + c, v);
    if (c == 0 && ld > D) store_tail(dop, plane, at + D, -dot);
  }
  if (c == 0 && row < nd_ld) ndelta[(long long)head * nd_ld + row] = row < nq ? -dot : 0.f;
}

}  // namespace f32
