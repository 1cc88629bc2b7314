// Fused primal (+ tangent) attention forward for fp32 on the Blackwell tensor cores.  Every product is six bf16 MMAs on
// three parts of its operands (f32_tc5_common.cuh).
//
// CTA = one 128-row query tile of one (batch, head), 384 threads:
//   warp 0        TMA producer (one lane), owner of the TMEM allocation
//   warp 1        MMA issuer (converged, one elected lane)
//   warps 4..11   two warpgroups; thread <-> query row <-> TMEM lane; group w takes the keys [32 w, 32 w + 32) of a tile in the
//                 softmax and half of the output columns in its registers
// Shared memory: the parts of Q and tQ (K-major, 128-byte swizzle), and a ring of 16 KiB units, each one part of two tiles of
// 64 rows x 64 columns: for the scores [K | tK] of 64 columns of D, for the outputs [V | tV] (D = 64) or the two halves of V or
// of tV (D = 128).  A unit is read by the products its part takes part in (lo: A hi; mid: A mid, hi; hi: A lo, mid, hi) and
// is free again; units stream in the order of the products, small parts first.  D = 128 with tangents: the lo part of Q is
// kept in TMEM (32 KiB of shared memory that the ring needs).
// TMEM: two score buffers [S | tS] (64 columns each), so that the scores of tile t + 1 are formed under the softmax of t;
// P and W = P * tS * scale, in three parts, go over the columns of S and tS they were made from, the lo parts to 64 columns
// beside them; one accumulator of 128 columns for the outputs of a tile.  A tensor core adds with truncation, so an accumulator
// never lives longer than one key tile: its columns are read back, rescaled and added in registers, rounded.
//
// What bounds it: the tensor pipe.  A 64-key tile at D = 128 with tangents is 168 instructions of 9984 cycles at the rates of
// mbar_wait_warp's comment, of 13600 measured; the rest are units that come late and the hand-overs of the one accumulator.
// Measured on a B200, B2 H8 L1024 D128, us, the register-tiled kernels / here with the splitting: O alone 297 / 73, with
// tangents 679 / 169, with an fp32 bias 721 / 181; D64 338 / 89, D32 169 / 71.  Error against 64 bits there: O 1.1e-6 -> 4.6e-7,
// tO 2.2e-6 -> 1.0e-6.
#include "f32_tc5_common.cuh"

namespace jvpfa {
namespace tc5 {

enum F32Mode : int { kPrimal = 0, kZeroTkv = 1, kDual = 2 };

template <int D_, int MODE>
struct FwdF32Cfg {
  static constexpr int D = D_;
  static constexpr int BM = 128, BN = 64;
  static constexpr bool DUAL = MODE != kPrimal;  // has tQ
  static constexpr bool TKV = MODE == kDual;     // has tK, tV
  static constexpr int SLOTS = MODE == kPrimal ? 3 : TKV ? 6 : 4;  // tensors in the workspace
  static constexpr int NSL = D > 64 ? 2 : 1;     // 64-column slices of D
  static constexpr int KS = D < 64 ? D / 16 : 4;  // contraction steps of a slice
  static constexpr int NTHREADS = 384;
  static constexpr int PART = BM * 128;           // one part of one slice of Q: 16 KiB
  static constexpr bool QLO_TMEM = D > 64 && DUAL;
  static constexpr int Q_PARTS = QLO_TMEM ? 2 : 3;
  static constexpr int UNIT_LOADS_S = TKV ? 2 : 1;
  // a unit of the scores: K and tK, 64 columns of one part; of the outputs: V and tV (D <= 64), two halves (D = 128)
  static constexpr int TILE = BN * 128;  // 8 KiB
  static constexpr int UNIT = (TKV || NSL == 2) ? 2 * TILE : TILE;
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_TQ = OFF_Q + NSL * Q_PARTS * PART;
  static constexpr int OFF_RING = OFF_TQ + (DUAL ? NSL * 3 * PART : 0);
  static constexpr int BUDGET = 227 * 1024 - 1024 - 1024 - 512;
  static constexpr int FIT = (BUDGET - OFF_RING) / UNIT;
  static constexpr int STAGES = FIT > 12 ? 12 : FIT;
  static_assert(STAGES >= 4, "ring");
  static constexpr int OFF_RED = OFF_RING + STAGES * UNIT;
  static constexpr int OFF_BAR = OFF_RED + 2 * BM * 4;
  static constexpr int SMEM_NEEDED = OFF_BAR + 512 + 1024;
  static constexpr int SMEM_BYTES = SMEM_NEEDED > 120 * 1024 ? SMEM_NEEDED : 120 * 1024;  // one CTA per SM: it allocates all of TMEM
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  // TMEM columns
  static constexpr int SC = 128;
  static constexpr int COL_LO = 2 * SC;   // lo parts of P and W
  static constexpr int COL_ACC = COL_LO + 64;
  static constexpr int COL_QLO = COL_ACC + 128;
  // outputs: pieces of at most 128 columns.  D <= 64: [O | tO'] ; D = 128: O, then tO'
  static constexpr int PIECES = (NSL == 2 && DUAL) ? 2 : 1;
  static constexpr int W_OUT = 32 * NSL;  // columns of O (and of tO') that a thread keeps
  static constexpr int N_SU = 3 * NSL;    // units of a tile's scores
};

// Slots of the tensors in the workspace
enum : int { kSlotQ = 0, kSlotK = 1, kSlotV = 2, kSlotTQ = 3, kSlotTK = 4, kSlotTV = 5 };

template <int D_, int MODE, int MK>
__global__ void __launch_bounds__(384, 1)
fwd_f32_tc5_kernel(const jvpfa_fwd_args a, const __grid_constant__ CUtensorMap map, const __nv_bfloat16* parts, int* status) {
  using C = FwdF32Cfg<D_, MODE>;
  constexpr int D = C::D, BM = C::BM, BN = C::BN, STAGES = C::STAGES, NSL = C::NSL, KS = C::KS;
  constexpr bool DUAL = C::DUAL, TKV = C::TKV;
  const bool dead_on_entry = *(volatile int*)(status + kF32GaveUp) != 0;

  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  float* red = reinterpret_cast<float*>(smem + C::OFF_RED);  // [2][BM]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* qlo_full = bars + 1;  // 256
  uint64_t* s_full = bars + 2;    // [2]
  uint64_t* p_full = bars + 4;    // [2], 256
  uint64_t* acc_full = bars + 6;
  uint64_t* acc_free = bars + 7;  // 256
  uint64_t* meet = bars + 8;      // [4], 64: the two warps of a quarter of the rows
  uint64_t* full = bars + 12;     // [STAGES]
  uint64_t* empty = full + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + STAGES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  const int BH = a.B * a.H;
  const int m0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * BM;  // heaviest causal tiles first
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL;
  int n_valid = L;
  if (a.mask.kind == JVPFA_MASK_KVLEN) {
    const int n = a.mask.kv_len[b];
    n_valid = n < 0 ? 0 : (n > L ? L : n);
  }
  const int n_end = causal ? min(n_valid, m0 + BM) : n_valid;
  const int n_tiles = (n_end + BN - 1) / BN;

  auto poison = [&]() {
    if (tid < BM && m0 + tid < L) a.lse[(size_t)bh * L + m0 + tid] = poison_f32();
  };
  if (dead_on_entry) {
    poison();
    return;
  }

  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(qlo_full, 256);
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_full + s, 256);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, 256);
    for (int s = 0; s < 4; ++s) mbar_init(meet + s, 64);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const AbortState ab{abort_flag, status};

  // (128 threads x 96 registers down from the 168 of the launch are the 256 x 48 that the others go up)
  // (in the branches of the roles: ptxas holds code behind a join of the two to the smaller number)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0 && n_tiles > 0) {
        prefetch_tmap(&map);
        auto load = [&](unsigned char* dst, uint64_t* bar, int slot, int part, int x, int y) {
          tma_load_4d(dst, &map, bar, x, y, bh, slot * 3 + part);
        };
        mbar_expect_tx(q_full, (C::Q_PARTS + (DUAL ? 3 : 0)) * NSL * C::PART);
        for (int p = 0; p < 3; ++p)
          for (int s = 0; s < NSL; ++s)
            for (int r = 0; r < 2; ++r) {  // rows m0 + 64 r: beyond the tensor they read as zeros
              const int off = (p * NSL + s) * C::PART + r * C::TILE;
              if (p < C::Q_PARTS) load(smem + C::OFF_Q + off, q_full, kSlotQ, p, 64 * s, m0 + 64 * r);
              if constexpr (DUAL) load(smem + C::OFF_TQ + off, q_full, kSlotTQ, p, 64 * s, m0 + 64 * r);
            }
        int u = 0;
        bool ok = true;
        // one unit: n tiles of 8 KiB, the i-th from (slot_i, part, column x_i)
        auto unit = [&](int n, int part, int y, int slot0, int x0, int slot1, int x1) {
          if (!ok) return;
          const int st = u % STAGES;
          if (!(ok = mbar_wait_backoff<64>(empty + st, ((u / STAGES) & 1) ^ 1, ab, kAbortKvEmpty))) return;
          unsigned char* dst = smem + C::OFF_RING + st * C::UNIT;
          mbar_expect_tx(full + st, n * C::TILE);
          load(dst, full + st, slot0, part, x0, y);
          if (n > 1) load(dst + C::TILE, full + st, slot1, part, x1, y);
          ++u;
        };
        auto scores = [&](int t) {
          for (int p = 2; p >= 0; --p)
            for (int s = 0; s < NSL; ++s) unit(TKV ? 2 : 1, p, t * BN, kSlotK, 64 * s, kSlotTK, 64 * s);
        };
        scores(0);
        for (int t = 0; ok && t < n_tiles; ++t) {
          if (t + 1 < n_tiles) scores(t + 1);
          if constexpr (NSL == 1) {
            for (int p = 2; p >= 0; --p) unit(TKV ? 2 : 1, p, t * BN, kSlotV, 0, kSlotTV, 0);
          } else {
            for (int p = 2; p >= 0; --p) unit(2, p, t * BN, kSlotV, 0, kSlotV, 64);
            if constexpr (DUAL)
              for (int p = 2; p >= 0; --p) {
                unit(2, p, t * BN, kSlotV, 0, kSlotV, 64);
                if constexpr (TKV) unit(2, p, t * BN, kSlotTV, 0, kSlotTV, 64);
              }
          }
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer: a converged warp, one elected lane
      if (n_tiles > 0) {
        constexpr int F = Fmt<__nv_bfloat16>::kIdesc;
        constexpr uint32_t id64 = make_idesc(F, BM, 64, 0, 0), id128 = make_idesc(F, BM, 128, 0, 0);
        constexpr uint32_t id64t = make_idesc(F, BM, 64, 0, 1), id128t = make_idesc(F, BM, 128, 0, 1);  // B MN-major
        constexpr uint32_t kLoMN = (uint32_t)(C::TILE >> 4) << 16;  // 64-column chunks of an MN-major operand are TILE apart
        constexpr uint32_t PART16 = C::PART >> 4, UNIT16 = C::UNIT >> 4;
        constexpr uint32_t id_s = TKV ? id128 : id64;
        const uint32_t q_lo = kDescLo | (smem_u32(smem + C::OFF_Q) >> 4), tq_lo = kDescLo | (smem_u32(smem + C::OFF_TQ) >> 4);
        const uint32_t ring16 = smem_u32(smem + C::OFF_RING) >> 4;
        int st = 0;
        uint32_t ph = 0;
        bool ok = mbar_wait_warp(q_full, 0, ab, kAbortQFull);
        if (C::QLO_TMEM && ok) ok = mbar_wait_warp(qlo_full, 0, ab, kAbortQFull);
        auto acquire = [&]() -> bool {
          if (!mbar_wait_warp(full + st, ph, ab, kAbortKvFull)) return ok = false;
          tc_fence_after();
          return true;
        };
        auto release = [&]() {  // (called by the elected lane)
          tc_commit(empty + st);
        };
        auto next = [&]() {
          if (++st == STAGES) st = 0, ph ^= 1;
        };
        // The scores of tile t: units of parts lo, mid, hi; part p of K meets the parts pa <= 2 - p of Q (tQ), small ones first.
        auto scores = [&](int t) {
          const uint32_t sc = tmem + (t & 1) * C::SC;
  #pragma unroll
          for (int p = 2; p >= 0; --p) {
  #pragma unroll
            for (int s = 0; s < NSL; ++s) {
              if (!acquire()) return;
              const uint32_t bk = kDescLo | (ring16 + st * UNIT16);
              if (elect_one()) {
  #pragma unroll
                for (int pa = 2 - p; pa >= 0; --pa) {
                  const uint32_t off = (pa * NSL + s) * PART16;
                  const bool first = p == 2 && s == 0;  // (pa = 0 then)
  #pragma unroll
                  for (int ks = 0; ks < KS; ++ks) {
                    if (C::QLO_TMEM && pa == 2)
                      umma_ts_lo<true>(sc, tmem + C::COL_QLO + s * 32 + ks * 8, bk + ks * 2, id_s);
                    else if (first && ks == 0)
                      umma_ss_lo<false>(sc, q_lo + off, bk, id_s);
                    else
                      umma_ss_lo<true>(sc, q_lo + off + ks * 2, bk + ks * 2, id_s);
                  }
                  if constexpr (DUAL) {
  #pragma unroll
                    for (int ks = 0; ks < KS; ++ks) {
                      if (!TKV && first && ks == 0)
                        umma_ss_lo<false>(sc + 64, tq_lo + off, bk, id64);
                      else
                        umma_ss_lo<true>(sc + 64, tq_lo + off + ks * 2, bk + ks * 2, id64);
                    }
                  }
                }
                release();
                if (p == 0 && s == NSL - 1) tc_commit(s_full + (t & 1));
              }
              next();
            }
          }
        };
        int piece = 0;
        // acc (+)= part pa of P (W) x the unit: contraction step kk = 16 keys
        auto outer = [&](uint32_t acc_col, uint32_t sc, bool w, int pa, uint32_t bm, uint32_t id, bool fresh) {
  #pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const uint32_t acol = pa < 2 ? sc + (w ? 64 : 0) + 8 * pa + 16 * kk
                                         : tmem + C::COL_LO + (w ? 16 : 0) + 32 * (kk >> 1) + 8 * (kk & 1);
            if (fresh && kk == 0)
              umma_ts_lo<false>(tmem + acc_col, acol, bm, id);
            else
              umma_ts_lo<true>(tmem + acc_col, acol, bm + kk * 128, id);
          }
        };
        auto begin_piece = [&]() -> bool {
          if (piece > 0 && !mbar_wait_warp(acc_free, (piece - 1) & 1, ab, kAbortOFull)) return ok = false;
          tc_fence_after();
          ++piece;
          return true;
        };
        auto outputs = [&](int t) {
          const uint32_t sc = tmem + (t & 1) * C::SC;
          if (!mbar_wait_warp(p_full + (t & 1), (t >> 1) & 1, ab, kAbortPFull) || !begin_piece()) {
            ok = false;
            return;
          }
  #pragma unroll
          for (int p = 2; p >= 0; --p) {  // D <= 64: [O | tO'] += P [V | tV], tO' += W V ; D = 128: O += P V
            if (!acquire()) return;
            const uint32_t bm = kLoMN | (ring16 + st * UNIT16);
            if (elect_one()) {
  #pragma unroll
              for (int pa = 2 - p; pa >= 0; --pa) {
                outer(C::COL_ACC, sc, false, pa, bm, TKV || NSL == 2 ? id128t : id64t, p == 2);
                if constexpr (DUAL && NSL == 1) outer(C::COL_ACC + 64, sc, true, pa, bm, id64t, !TKV && p == 2);
              }
              release();
              if (p == 0) tc_commit(acc_full);
            }
            next();
          }
          if constexpr (DUAL && NSL == 2) {
            if (!begin_piece()) return;
  #pragma unroll
            for (int p = 2; p >= 0; --p) {  // tO' += W V + P tV
  #pragma unroll
              for (int x = 0; x < (TKV ? 2 : 1); ++x) {
                if (!acquire()) return;
                const uint32_t bm = kLoMN | (ring16 + st * UNIT16);
                if (elect_one()) {
  #pragma unroll
                  for (int pa = 2 - p; pa >= 0; --pa) outer(C::COL_ACC, sc, x == 0, pa, bm, id128t, p == 2 && x == 0);
                  release();
                  if (p == 0 && x == (TKV ? 1 : 0)) tc_commit(acc_full);
                }
                next();
              }
            }
          }
        };
        if (ok) scores(0);
        for (int t = 0; ok && t < n_tiles; ++t) {
          if (t + 1 < n_tiles) scores(t + 1);
          if (ok) outputs(t);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------ softmax, outputs
    const int w = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int i = m0 + row;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const float scale_log2 = a.sm_scale * kLog2e;
    if constexpr (C::QLO_TMEM) {
      // the lo part of this row of Q, columns [64 w, 64 w + 64), to its 32 TMEM columns
      uint32_t r[32];
      const uint4* src = reinterpret_cast<const uint4*>(
          parts + ((size_t)(kSlotQ * 3 + 2) * BH + bh) * L * D + (size_t)min(i, L - 1) * D + 64 * w);
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint4 v = i < L ? ldg_nc_v4(src + x) : make_uint4(0u, 0u, 0u, 0u);
        r[4 * x] = v.x, r[4 * x + 1] = v.y, r[4 * x + 2] = v.z, r[4 * x + 3] = v.w;
      }
      tmem_st32(tmem + lane_off + C::COL_QLO + 32 * w, r);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(qlo_full);
    }
    const F32RowMask<MK> rm(a.mask, a.mask_bits, b, h, a.H, i, L);
    // Causal: whether V or tV holds what is not finite up to the last key of this tile, block by block of the splitting pass.
    const long long plane = (long long)BH * L * D, n_blocks = (plane + kSplitBlock - 1) / kSplitBlock;
    const uint32_t* found = reinterpret_cast<const uint32_t*>(parts + C::SLOTS * 3 * plane);
    const long long block0 = (long long)bh * L * D / kSplitBlock, block1 = ((long long)bh * L + min(L, m0 + BM)) * D / kSplitBlock;
    bool any_found = false;
    if (MK == 0 && causal) {
      for (long long x = block0 + lane; x <= min(block1, n_blocks - 1); x += 32)
        any_found = any_found || found[x] != 0u || (TKV && found[n_blocks + x] != 0u);
      any_found = __any_sync(0xffffffffu, any_found);
    }
    float acc_o[C::W_OUT], acc_t[DUAL ? C::W_OUT : 1];
#pragma unroll
    for (int x = 0; x < C::W_OUT; ++x) {
      acc_o[x] = 0.f;
      if constexpr (DUAL) acc_t[x] = 0.f;
    }
    float m_used = -INFINITY, l_run = 0.f, mu_run = 0.f;
    int piece = 0;
    bool alive = true;
    // What the mask holds for a tile's keys.  Requested a tile ahead, once this one's probabilities are written: it arrives under
    // the output products.  (Behind the last tile that tile's again: under a condition this one's would have to be kept.)
    float bias[MK == 2 ? 32 : 1];
    uint32_t next_live = 0u;
    auto fetch_mask = [&](int t) {
      const int n0 = min(t, n_tiles - 1) * BN + 32 * w;
      int hi = min(32, n_valid - n0);  // live keys of this row among the 32: a bit each
      if (causal) hi = min(hi, i - n0 + 1);
      next_live = rm.fetch(n0, first_columns(hi), bias);
    };
    if (n_tiles > 0) fetch_mask(0);
    for (int t = 0; alive && t < n_tiles; ++t) {
      const uint32_t tS = tmem + lane_off + (t & 1) * C::SC + 32 * w, tTS = tS + 64;
      const uint32_t tLO = tmem + lane_off + C::COL_LO + 32 * w;
      const uint32_t live = next_live;
      if (!mbar_wait(s_full + (t & 1), (t >> 1) & 1, ab, kAbortSFull)) {
        alive = false;
        break;
      }
      tc_fence_after();
      float mx = -INFINITY;
      {
        uint32_t x[32];
        tmem_ld32(tS, x);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          float v = f32_score<MK>(__uint_as_float(x[c]), scale_log2, MK == 2 ? bias[c] : 0.f);
          if (!((live >> c) & 1u)) v = -INFINITY;
          x[c] = __float_as_uint(v);
          mx = fmaxf(mx, v);
        }
        tmem_st32(tS, x);  // scaled, biased and masked, for the second pass
      }
      // the row's maximum over both halves of the tile
      red[w * BM + row] = mx;
      mbar_arrive(meet + quarter);
      if (!mbar_wait(meet + quarter, t & 1, ab, kAbortAux)) {
        alive = false;
        break;
      }
      mx = fmaxf(mx, red[(w ^ 1) * BM + row]);
      // The running maximum itself is the reference: P is at most 1, so nothing overflows before the result does.  (A reference up
      // to 2^8 below it, as in the 16-bit kernels, saves nothing here: alpha goes into the additions below in any case.)
      float alpha = 1.f;
      if (mx > m_used) {
        alpha = fast_exp2(m_used - mx);
        m_used = mx;
      }
      const float m_eff = m_used == -INFINITY ? 0.f : m_used;
      l_run *= alpha, mu_run *= alpha;
      tmem_wait_st();
      float ls = 0.f, ms = 0.f;
#pragma unroll
      for (int s = 0; s < 2; ++s) {  // 16 keys at a time: one contraction step of the output products
        uint32_t x[16], y[DUAL ? 16 : 1];
        tmem_ld16(tS + 16 * s, x);
        if constexpr (DUAL) tmem_ld16(tTS + 16 * s, y);
        tmem_wait_ld();
        uint32_t ph[16], pl[8];  // hi parts, then mid parts ; lo parts
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float p0 = fast_exp2(__uint_as_float(x[2 * c]) - m_eff), p1 = fast_exp2(__uint_as_float(x[2 * c + 1]) - m_eff);
          ls += p0 + p1;
          split3_pair(p0, p1, ph[c], ph[8 + c], pl[c]);
          if constexpr (DUAL) {
            // (a masked key's tangent score does not count, whatever it is)
            const float t0 = (live >> (16 * s + 2 * c)) & 1u ? __uint_as_float(y[2 * c]) : 0.f;
            const float t1 = (live >> (16 * s + 2 * c + 1)) & 1u ? __uint_as_float(y[2 * c + 1]) : 0.f;
            const float w0 = p0 * (t0 * a.sm_scale), w1 = p1 * (t1 * a.sm_scale);
            ms += w0 + w1;
            y[2 * c] = __float_as_uint(w0), y[2 * c + 1] = __float_as_uint(w1);
          }
        }
        tmem_st16(tS + 16 * s, ph);
        tmem_st8(tLO + 8 * s, pl);
        if constexpr (DUAL) {
#pragma unroll
          for (int c = 0; c < 8; ++c) split3_pair(__uint_as_float(y[2 * c]), __uint_as_float(y[2 * c + 1]), ph[c], ph[8 + c], pl[c]);
          tmem_st16(tTS + 16 * s, ph);
          tmem_st8(tLO + 16 + 8 * s, pl);
        }
      }
      l_run += ls, mu_run += ms;
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full + (t & 1));
      fetch_mask(t + 1);
      // The tile's outputs: read back, rescaled and added with rounding.
#pragma unroll
      for (int pc = 0; pc < C::PIECES; ++pc) {
        if (!mbar_wait(acc_full, piece & 1, ab, kAbortOFull)) {
          alive = false;
          break;
        }
        ++piece;
        tc_fence_after();
        const uint32_t tA = tmem + lane_off + C::COL_ACC;
        auto add = [&](float* acc, uint32_t col) {
          uint32_t r[32];
          tmem_ld32(col, r);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 32; ++c) acc[c] = __fmaf_rn(acc[c], alpha, __uint_as_float(r[c]));
        };
        if constexpr (NSL == 1) {
          add(acc_o, tA + 32 * w);
          if constexpr (DUAL) add(acc_t, tA + 64 + 32 * w);
        } else if (pc == 0) {
          add(acc_o, tA + 64 * w);
          add(acc_o + 32, tA + 64 * w + 32);
        } else {
          if constexpr (DUAL) {
            add(acc_t, tA + 64 * w);
            add(acc_t + 32, tA + 64 * w + 32);
          }
        }
        tc_fence_before();
        mbar_arrive(acc_free);
      }
    }
    // ---- epilogue: the two halves of a row's sums, then O = acc/l, tO = acc'/l - (mu/l) O, lse = m + log2 l
    if (alive) {
      float* sums = reinterpret_cast<float*>(smem + C::OFF_RING);  // [2][2][BM]: the ring is idle
      sums[w * BM + row] = l_run;
      sums[(2 + w) * BM + row] = mu_run;
      mbar_arrive(meet + quarter);
      if (mbar_wait(meet + quarter, n_tiles & 1, ab, kAbortAux)) {
        l_run = sums[row] + sums[BM + row];
        mu_run = sums[2 * BM + row] + sums[3 * BM + row];
        const bool none = !(l_run > 0.f);  // no key, or what is not a number: sums of zeros stay zeros, and NaN stays NaN
        const float inv_l = none ? 0.f : 1.f / l_run;
        const float mu = mu_run * inv_l;
        if (i < L) {
          if (w == 0) {
            a.lse[(size_t)bh * L + i] = none ? INFINITY : m_used + log2f(l_run);
            if constexpr (DUAL) a.mu[(size_t)bh * L + i] = mu;
          }
          if (D > 32 || w == 0) {
            if constexpr (MK == 0) {
              if (any_found) {  // the columns in which a key that this row attends is not finite
                const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
                const long long row_stride = strided ? a.in_stride[2] : D;
                const long long head = (strided ? b * a.in_stride[0] + h * a.in_stride[1] : (long long)bh * L * D) + C::W_OUT * w;
                for (long long x = block0; x <= min(block1, n_blocks - 1); ++x) {
                  if (found[x] == 0u && !(TKV && found[n_blocks + x] != 0u)) continue;
                  const long long first = x * kSplitBlock / D - (long long)bh * L, end = min((long long)i + 1, first + kSplitBlock / D);
                  for (long long j = max(first, 0ll); j < end; ++j) {
#pragma unroll
                    for (int c = 0; c < C::W_OUT; ++c) {
                      if (!isfinite(reinterpret_cast<const float*>(a.v)[head + j * row_stride + c])) {
                        acc_o[c] = poison_f32();
                        if constexpr (DUAL) acc_t[c] = poison_f32();
                      }
                      if constexpr (TKV)
                        if (!isfinite(reinterpret_cast<const float*>(a.tv)[head + j * row_stride + c])) acc_t[c] = poison_f32();
                    }
                  }
                }
              }
            }
            float4* po = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.o) + ((size_t)bh * L + i) * D + C::W_OUT * w);
            float4* pt = DUAL ? reinterpret_cast<float4*>(reinterpret_cast<float*>(a.to) + ((size_t)bh * L + i) * D + C::W_OUT * w) : nullptr;
#pragma unroll
            for (int c = 0; c < C::W_OUT / 4; ++c) {
              float o[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) o[e] = acc_o[4 * c + e] * inv_l;
              po[c] = make_float4(o[0], o[1], o[2], o[3]);
              if constexpr (DUAL) {
                float u[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) u[e] = acc_t[4 * c + e] * inv_l - mu * o[e];
                pt[c] = make_float4(u[0], u[1], u[2], u[3]);
              }
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    poison();
    if (tid == 0) *(volatile int*)(status + kF32GaveUp) = *abort_flag;
  }
  if (warp == 0) {
    if (*abort_flag != 0) {
      // Something gave up: give copies and MMAs that may still be in flight time to land before the TMEM
      // columns go back to the allocator.
      const long long t0 = clock64();
      while (clock64() - t0 < (1ll << 22)) {
      }
    }
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---- the parts of the inputs ----------------------------------------------------------------------------------------
// Eight elements of a row per thread.
__global__ void __launch_bounds__(256) split3_kernel(const SplitArgs s) {
  const long long e = (long long)blockIdx.x * kSplitBlock + threadIdx.x * 8;
  const int slot = blockIdx.y;
  const bool clean = (s.clean >> slot) & 1u;
  bool found = false;
  if (e < s.plane) {
    const long long row = e / s.D;
    const int col = (int)(e - row * s.D);
    const long long bh = row / s.L;
    const int i = (int)(row - bh * s.L);
    float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
    if (s.kv_len == nullptr || !((s.padded >> slot) & 1u) || i < s.kv_len[bh / s.H]) {
      const float4* src = reinterpret_cast<const float4*>(s.src[slot] + (bh / s.H) * s.st[slot][0] + (bh % s.H) * s.st[slot][1] +
                                                          (long long)i * s.st[slot][2] + col);
      x0 = __ldg(src), x1 = __ldg(src + 1);
    }
    float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    if (clean) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (!isfinite(x[c])) found = true, x[c] = 0.f;
    }
    uint32_t r[3][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float h[2], m[2], l[2];
      split3(x[2 * c], h[0], m[0], l[0]);
      split3(x[2 * c + 1], h[1], m[1], l[1]);
      r[0][c] = pack_bf16(h[0], h[1]), r[1][c] = pack_bf16(m[0], m[1]), r[2][c] = pack_bf16(l[0], l[1]);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint4*>(s.dst + ((long long)slot * 3 + p) * s.plane + e) = make_uint4(r[p][0], r[p][1], r[p][2], r[p][3]);
  }
  if (clean && s.found != nullptr) {
    const int any = __syncthreads_or(found);
    if (threadIdx.x == 0) s.found[__popc(s.clean & ((1u << slot) - 1u)) * gridDim.x + blockIdx.x] = any;
  }
}

int launch_split3(const SplitArgs& s, int slots, cudaStream_t stream) {
  const dim3 grid((unsigned)((s.plane + kSplitBlock - 1) / kSplitBlock), slots);
  split3_kernel<<<grid, 256, 0, stream>>>(s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch split3");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <int D, int MODE, int MK>
static int launch_fwd_f32(const jvpfa_fwd_args& a, const CUtensorMap& map, int* status, cudaStream_t stream) {
  using C = FwdF32Cfg<D, MODE>;
  auto kern = fwd_f32_tc5_kernel<D, MODE, MK>;
  static SmemOptIn opt_in;
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return JVPFA_ERR_CUDA;
  const dim3 grid((a.L + C::BM - 1) / C::BM, a.B * a.H);
  kern<<<grid, C::NTHREADS, C::SMEM_BYTES, stream>>>(a, map, static_cast<const __nv_bfloat16*>(a.workspace), status);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch fwd_f32_tc5");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <int D, int MODE>
static int launch_fwd_f32_mask(const jvpfa_fwd_args& a, const CUtensorMap& map, int* status, cudaStream_t s) {
  if (a.mask.kind == JVPFA_MASK_BOOL) return launch_fwd_f32<D, MODE, 1>(a, map, status, s);
  if (a.mask.kind == JVPFA_MASK_BIAS) return launch_fwd_f32<D, MODE, 2>(a, map, status, s);
  return launch_fwd_f32<D, MODE, 0>(a, map, status, s);
}

template <int D>
static int launch_fwd_f32_mode(const jvpfa_fwd_args& a, const CUtensorMap& map, int* status, cudaStream_t s) {
  if (!a.tq) return launch_fwd_f32_mask<D, kPrimal>(a, map, status, s);
  if (a.flags & JVPFA_ZERO_TKV) return launch_fwd_f32_mask<D, kZeroTkv>(a, map, status, s);
  return launch_fwd_f32_mask<D, kDual>(a, map, status, s);
}

}  // namespace tc5

static int fwd_f32_slots(const jvpfa_fwd_args& a) { return !a.tq ? 3 : (a.flags & JVPFA_ZERO_TKV) ? 4 : 6; }

long long fwd_f32_tc5_workspace(const jvpfa_fwd_args& a) {
  if (a.dtype != JVPFA_FP32 || a.impl == JVPFA_IMPL_GENERIC) return 0;
  if (a.impl == JVPFA_IMPL_AUTO && !tc5::f32_rows_enough(a.mask, a.B, a.H, a.L, a.D)) return 0;
  const long long plane = (long long)a.B * a.H * a.L * a.D, blocks = (plane + tc5::kSplitBlock - 1) / tc5::kSplitBlock;
  return fwd_f32_slots(a) * 3 * 2 * plane + (a.mask.kind == JVPFA_MASK_CAUSAL ? 2 * 4 * blocks : 0);
}

bool fwd_f32_tc5_eligible(const jvpfa_fwd_args& a) {
  const long long need = fwd_f32_tc5_workspace(a);
  return need > 0 && a.workspace != nullptr && a.workspace_bytes >= need && (reinterpret_cast<uintptr_t>(a.workspace) & 15u) == 0;
}

int launch_fwd_f32_tc5(const jvpfa_fwd_args& a, cudaStream_t stream) {
  using namespace tc5;
  int* status = tc5_status_device_ptr();
  if (!status) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  const int slots = fwd_f32_slots(a);
  SplitArgs s{};
  s.dst = static_cast<__nv_bfloat16*>(a.workspace);
  s.plane = (long long)a.B * a.H * a.L * a.D;
  s.H = a.H, s.L = a.L, s.D = a.D;
  if (a.mask.kind == JVPFA_MASK_KVLEN) {
    s.kv_len = a.mask.kv_len;
    s.padded = 1u << kSlotK | 1u << kSlotV | 1u << kSlotTK | 1u << kSlotTV;
  }
  if (a.mask.kind == JVPFA_MASK_CAUSAL) {
    s.clean = 1u << kSlotV | (slots == 6 ? 1u << kSlotTV : 0u);
    s.found = reinterpret_cast<uint32_t*>(s.dst + slots * 3 * s.plane);
  }
  const void* src[kF32MaxSlots] = {a.q, a.k, a.v, a.tq, a.tk, a.tv};
  for (int n = 0; n < slots; ++n) s.set(n, src[n], a.in_stride);
  CUtensorMap map;
  if (!encode_map_parts(&map, a.workspace, a.D, a.L, a.B * a.H, slots * 3)) {
    set_last_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled(fwd f32)");
    return JVPFA_ERR_CUDA;
  }
  const int rc = launch_split3(s, slots, stream);
  if (rc) return rc;
  if (a.D == 32) return launch_fwd_f32_mode<32>(a, map, status, stream);
  if (a.D == 64) return launch_fwd_f32_mode<64>(a, map, status, stream);
  return launch_fwd_f32_mode<128>(a, map, status, stream);
}

}  // namespace jvpfa
