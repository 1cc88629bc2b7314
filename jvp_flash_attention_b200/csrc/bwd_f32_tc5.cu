// Backward for fp32 on the Blackwell tensor cores, every product as six bf16 MMAs on three parts of its operands
// (f32_tc5_common.cuh): through O, and dQ alone through tO where K and V have no tangents (the second differentiation of a
// Hessian-vector product along q).
//     S = Q K^T,  P = 2^(scale S + bias - lse)
//     through O   gS = P (gO V^T - delta),  dV = P^T gO,  dK = scale gS^T Q
//     through tO  tS = tQ K^T, E = G V^T,  gS = P (E (tS - mu) - eps tS - cterm)
//     dQ = scale gS K
// in two launches, one that owns queries (dQ) and one that owns keys (dK, dV), as the register-tiled kernels.
//
// The launch that owns queries: CTA = one 128-row query tile of one (batch, head), 384 threads with the roles of the forward
// (fwd_f32_tc5.cu): producer, issuing warp, two elementwise warpgroups (thread <-> query row <-> TMEM lane; group w takes keys
// [32 w, 32 w + 32) of a 64-key tile, and half of dQ's columns in its registers).
// Shared memory: the parts of the own operands (Q, gO | Q, tQ, G), and a ring of 8 KiB units: one part of 64 keys x 64 columns of
// K, of V, and of K once more for dQ.  D = 128: the lo parts of the own operands are TMEM operands.
// TMEM: the scores of a tile (two buffers where they fit: the next tile's are formed under this one's elementwise work); gS in
// three parts over the columns it was made from; one accumulator for a tile's dQ, read back and added in registers.
//
// Bound by the tensor pipe as the forward.  Measured on a B200, B2 H8 L1024, us, the register-tiled kernels / here with the
// splitting: dQ through O D128 353 / 103, D64 197 / 58, D32 125 / 44; dQ through tO 566 / 142, 298 / 73, 144 / 52; all three
// gradients through O 853 / 248, 468 / 125, 282 / 102.
#include "f32_tc5_common.cuh"

namespace jvpfa {
namespace tc5 {

template <int D_, bool GT_>
struct DqF32Cfg {
  static constexpr int D = D_;
  static constexpr bool GT = GT_;  // through tO; otherwise through O
  static constexpr int BM = 128, BN = 64;
  static constexpr int NSL = D > 64 ? 2 : 1;
  static constexpr int KS = D < 64 ? D / 16 : 4;
  static constexpr int NTHREADS = 384;
  static constexpr int NA = GT ? 3 : 2;  // Q, gO | Q, tQ, G
  static constexpr int OP_X = NA - 1;    // the operand that meets V
  static constexpr bool LO_TMEM = D > 64;
  static constexpr int A_PARTS = LO_TMEM ? 2 : 3;
  static constexpr int PART = BM * 128;  // one part of one 64-column slice of an own operand
  static constexpr int TILE = BN * 128;  // a unit of the ring
  static constexpr int OFF_RING = NA * A_PARTS * NSL * PART;
  static constexpr int BUDGET = 227 * 1024 - 1024 - 512;
  static constexpr int FIT = (BUDGET - OFF_RING) / TILE;
  static constexpr int STAGES = FIT > 16 ? 16 : FIT;
  static_assert(STAGES >= 4, "ring");
  static constexpr int OFF_BAR = OFF_RING + STAGES * TILE;
  static constexpr int SMEM_NEEDED = OFF_BAR + 512 + 1024;
  static constexpr int SMEM_BYTES = SMEM_NEEDED > 120 * 1024 ? SMEM_NEEDED : 120 * 1024;  // one CTA per SM: it allocates all of TMEM
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  // TMEM columns: score buffers [S | (tS) | X], X = gO V^T or E
  static constexpr int SC = 64 * NA;
  static constexpr int COL_TS = 64, COL_X = SC - 64;
  static constexpr int NBUF = LO_TMEM && GT ? 1 : 2;
  static constexpr int COL_LO = NBUF * SC;
  static constexpr int COL_ACC = COL_LO + (LO_TMEM ? NA * 32 * NSL : 0);
  static_assert(COL_ACC + 64 * NSL <= 512, "TMEM");
  static constexpr int W_OUT = 32 * NSL;  // columns of dQ that a thread keeps
};

enum : int { kDqSlotQ = 0, kDqSlotK = 1, kDqSlotV = 2, kDqSlotA = 3, kDqSlotB = 4 };  // A: gO, or tQ with G in B

template <int D_, bool GT_, int MK>
__global__ void __launch_bounds__(384, 1)
bwd_f32_dq_kernel(const jvpfa_bwd_args a, const __grid_constant__ CUtensorMap map, const __nv_bfloat16* parts, int* status) {
  using C = DqF32Cfg<D_, GT_>;
  constexpr int D = C::D, BM = C::BM, BN = C::BN, STAGES = C::STAGES, NSL = C::NSL, KS = C::KS, NA = C::NA, NBUF = C::NBUF;
  constexpr bool GT = C::GT;
  const bool dead_on_entry = *(volatile int*)(status + kF32GaveUp) != 0;

  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* a_full = bars + 0;
  uint64_t* alo_full = bars + 1;  // 256
  uint64_t* s_full = bars + 2;    // [NBUF]
  uint64_t* p_full = bars + 4;    // [NBUF], 256
  uint64_t* acc_full = bars + 6;
  uint64_t* acc_free = bars + 7;  // 256
  uint64_t* full = bars + 8;      // [STAGES]
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
    if (tid < BM && m0 + tid < L) poison_row<float>(a.dq, (size_t)bh * L + m0 + tid, D);
  };
  if (dead_on_entry) {
    poison();
    return;
  }

  if (tid == 0) {
    mbar_init(a_full, 1);
    mbar_init(alo_full, 256);
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_full + s, 256);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, 256);
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

  // (128 threads x 96 registers down from the 168 of the launch are the 256 x 48 that the others go up; in the branches of the
  // roles, because ptxas holds code behind a join of the two to the smaller number)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0 && n_tiles > 0) {
        prefetch_tmap(&map);
        auto load = [&](unsigned char* dst, uint64_t* bar, int slot, int part, int x, int y) {
          tma_load_4d(dst, &map, bar, x, y, bh, slot * 3 + part);
        };
        mbar_expect_tx(a_full, NA * C::A_PARTS * NSL * C::PART);
        for (int op = 0; op < NA; ++op) {
          const int slot = op == 0 ? kDqSlotQ : op == 1 ? kDqSlotA : kDqSlotB;
          for (int p = 0; p < C::A_PARTS; ++p)
            for (int s = 0; s < NSL; ++s)
              for (int r = 0; r < 2; ++r)  // rows m0 + 64 r: beyond the tensor they read as zeros
                load(smem + ((op * C::A_PARTS + p) * NSL + s) * C::PART + r * C::TILE, a_full, slot, p, 64 * s, m0 + 64 * r);
        }
        int st = 0;
        uint32_t ph = 1;
        bool ok = true;
        auto units = [&](int t, int slot) {  // one part and slice after another, the lo parts first
          for (int p = 2; p >= 0; --p)
            for (int s = 0; s < NSL; ++s) {
              if (!ok || !(ok = mbar_wait_backoff<64>(empty + st, ph, ab, kAbortBwdLoopEmpty))) return;
              mbar_expect_tx(full + st, C::TILE);
              load(smem + C::OFF_RING + st * C::TILE, full + st, slot, p, 64 * s, t * BN);
              if (++st == STAGES) st = 0, ph ^= 1;
            }
        };
        auto scores = [&](int t) { units(t, kDqSlotK), units(t, kDqSlotV); };
        if (NBUF == 2) scores(0);
        for (int t = 0; ok && t < n_tiles; ++t) {
          if (NBUF == 1)
            scores(t);
          else if (t + 1 < n_tiles)
            scores(t + 1);
          units(t, kDqSlotK);
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer: a converged warp, one elected lane
      if (n_tiles > 0) {
        constexpr int F = Fmt<__nv_bfloat16>::kIdesc;
        constexpr uint32_t id64 = make_idesc(F, BM, 64, 0, 0), id64t = make_idesc(F, BM, 64, 0, 1);  // B K-major, MN-major
        constexpr uint32_t kLoMN = (uint32_t)(C::TILE >> 4) << 16;  // (one 64-column chunk: the leading offset is not used)
        constexpr uint32_t PART16 = C::PART >> 4, TILE16 = C::TILE >> 4;
        const uint32_t a_lo = kDescLo | (smem_u32(smem) >> 4);
        const uint32_t ring16 = smem_u32(smem + C::OFF_RING) >> 4;
        int st = 0;
        uint32_t ph = 0;
        bool ok = mbar_wait_warp(a_full, 0, ab, kAbortBwdOwn);
        if (C::LO_TMEM && ok) ok = mbar_wait_warp(alo_full, 0, ab, kAbortBwdOwn);
        auto acquire = [&]() -> bool {
          if (!mbar_wait_warp(full + st, ph, ab, kAbortBwdLoopFull)) return ok = false;
          tc_fence_after();
          return true;
        };
        auto next = [&]() {
          if (++st == STAGES) st = 0, ph ^= 1;
        };
        // col (+)= part pa of own operand op, slice s, x the unit at bk
        auto score = [&](uint32_t col, int op, int pa, int s, uint32_t bk, bool first) {
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) {
            if (C::LO_TMEM && pa == 2)
              umma_ts_lo<true>(col, tmem + C::COL_LO + (op * NSL + s) * 32 + ks * 8, bk + ks * 2, id64);
            else if (first && ks == 0)
              umma_ss_lo<false>(col, a_lo + ((op * C::A_PARTS + pa) * NSL + s) * PART16, bk, id64);
            else
              umma_ss_lo<true>(col, a_lo + ((op * C::A_PARTS + pa) * NSL + s) * PART16 + ks * 2, bk + ks * 2, id64);
          }
        };
        auto scores = [&](int t) {
          const uint32_t sc = tmem + (t % NBUF) * C::SC;
#pragma unroll
          for (int side = 0; side < 2; ++side) {  // K, then V
#pragma unroll
            for (int p = 2; p >= 0; --p) {
#pragma unroll
              for (int s = 0; s < NSL; ++s) {
                if (!acquire()) return;
                const uint32_t bk = kDescLo | (ring16 + st * TILE16);
                if (elect_one()) {
#pragma unroll
                  for (int pa = 2 - p; pa >= 0; --pa) {  // small products first
                    const bool first = p == 2 && s == 0;
                    if (side == 0) {
                      score(sc, 0, pa, s, bk, first);
                      if constexpr (GT) score(sc + C::COL_TS, 1, pa, s, bk, first);
                    } else {
                      score(sc + C::COL_X, C::OP_X, pa, s, bk, first);
                    }
                  }
                  tc_commit(empty + st);
                  if (side == 1 && p == 0 && s == NSL - 1) tc_commit(s_full + t % NBUF);
                }
                next();
              }
            }
          }
        };
        auto outputs = [&](int t) {
          const uint32_t sc = tmem + (t % NBUF) * C::SC;
          if (!mbar_wait_warp(p_full + t % NBUF, (t / NBUF) & 1, ab, kAbortBwdPFull) ||
              (t > 0 && !mbar_wait_warp(acc_free, (t - 1) & 1, ab, kAbortBwdDone))) {
            ok = false;
            return;
          }
#pragma unroll
          for (int p = 2; p >= 0; --p) {
#pragma unroll
            for (int s = 0; s < NSL; ++s) {
              if (!acquire()) return;
              const uint32_t bm = kLoMN | (ring16 + st * TILE16);
              if (elect_one()) {
#pragma unroll
                for (int pa = 2 - p; pa >= 0; --pa) {
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk) {  // 16 keys
                    const uint32_t acol = sc + (pa < 2 ? 8 * pa : C::COL_X) + 16 * kk;
                    if (p == 2 && kk == 0)
                      umma_ts_lo<false>(tmem + C::COL_ACC + 64 * s, acol, bm, id64t);
                    else
                      umma_ts_lo<true>(tmem + C::COL_ACC + 64 * s, acol, bm + kk * 128, id64t);
                  }
                }
                tc_commit(empty + st);
                if (p == 0 && s == NSL - 1) tc_commit(acc_full);
              }
              next();
            }
          }
        };
        if (NBUF == 2 && ok) scores(0);
        for (int t = 0; ok && t < n_tiles; ++t) {
          if (NBUF == 1)
            scores(t);  // (over the parts of gS of the tile before, whose products were issued before)
          else if (t + 1 < n_tiles)
            scores(t + 1);
          if (ok) outputs(t);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------ elementwise, dQ
    const int w = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int i = m0 + row;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const float scale = a.sm_scale, scale_log2 = a.sm_scale * kLog2e;
    if constexpr (C::LO_TMEM) {
      // the lo parts of this row of the own operands, columns [64 w, 64 w + 64), to their 32 TMEM columns each
#pragma unroll
      for (int op = 0; op < NA; ++op) {
        const int slot = op == 0 ? kDqSlotQ : op == 1 ? kDqSlotA : kDqSlotB;
        uint32_t r[32];
        const uint4* src =
            reinterpret_cast<const uint4*>(parts + ((size_t)(slot * 3 + 2) * BH + bh) * L * D + (size_t)min(i, L - 1) * D + 64 * w);
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const uint4 v = i < L ? ldg_nc_v4(src + x) : make_uint4(0u, 0u, 0u, 0u);
          r[4 * x] = v.x, r[4 * x + 1] = v.y, r[4 * x + 2] = v.z, r[4 * x + 3] = v.w;
        }
        tmem_st32(tmem + lane_off + C::COL_LO + (op * NSL + w) * 32, r);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(alo_full);
    }
    const F32RowMask<MK> rm(a.mask, a.mask_bits, b, h, a.H, i, L);
    const size_t stat = (size_t)bh * L + i;
    const float lse = i < L ? a.lse[stat] : INFINITY;
    float sub = i < L ? a.delta[stat] : 0.f, mu = 0.f, eps = 0.f;
    if (GT && i < L) sub += a.cterm[stat], mu = a.mu[stat], eps = a.eps[stat];
    float acc[C::W_OUT];
#pragma unroll
    for (int x = 0; x < C::W_OUT; ++x) acc[x] = 0.f;
    bool alive = true;
    // What the mask holds for a tile's keys, requested a tile ahead as in the forward.  (D = 128: at the tile's own beginning, where
    // the scores of one buffer are still being formed; 144 us through tO at B2 H8 L1024 with a bias, 158 ahead.)
    constexpr bool AHEAD = D < 128;
    float bias[MK == 2 ? 32 : 1];
    uint32_t live = 0u;
    auto fetch_mask = [&](int t) -> uint32_t {
      const int n0 = min(t, n_tiles - 1) * BN + 32 * w;
      int hi = min(32, n_valid - n0);  // live keys of this row among the 32: a bit each
      if (causal) hi = min(hi, i - n0 + 1);
      return rm.fetch(n0, first_columns(hi), bias);
    };
    uint32_t next_live = 0u;
    if (AHEAD && n_tiles > 0) next_live = fetch_mask(0);
    for (int t = 0; t < n_tiles; ++t) {
      const uint32_t tS = tmem + lane_off + (t % NBUF) * C::SC + 32 * w;
      live = AHEAD ? next_live : fetch_mask(t);
      if (!mbar_wait(s_full + t % NBUF, (t / NBUF) & 1, ab, kAbortBwdSFull)) {
        alive = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < 2; ++s) {  // 16 keys at a time: one contraction step of the dQ products
        uint32_t x[16], y[16], z[GT ? 16 : 1];
        tmem_ld16(tS + 16 * s, x);
        tmem_ld16(tS + C::COL_X + 16 * s, y);
        if constexpr (GT) tmem_ld16(tS + C::COL_TS + 16 * s, z);
        tmem_wait_ld();
        uint32_t gh[16], gl[8];  // hi parts, then mid parts ; lo parts
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          float g[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int n = 2 * c + e;
            const float v = f32_score<MK>(__uint_as_float(x[n]), scale_log2, MK == 2 ? bias[16 * s + n] : 0.f);
            const float p = fast_exp2(v - lse);
            float u = __uint_as_float(y[n]);
            if constexpr (GT) {
              const float ts = __uint_as_float(z[n]) * scale;
              u = u * (ts - mu) - eps * ts;
            }
            g[e] = (live >> (16 * s + n)) & 1u ? p * (u - sub) : 0.f;  // (nothing of a masked key counts, whatever it is)
          }
          split3_pair(g[0], g[1], gh[c], gh[8 + c], gl[c]);
        }
        tmem_st16(tS + 16 * s, gh);
        tmem_st8(tS + C::COL_X + 16 * s, gl);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full + t % NBUF);
      if constexpr (AHEAD) next_live = fetch_mask(t + 1);
      if (!mbar_wait(acc_full, t & 1, ab, kAbortBwdDone)) {
        alive = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int x = 0; x < NSL; ++x) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_off + C::COL_ACC + C::W_OUT * w + 32 * x, r);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[32 * x + c] += __uint_as_float(r[c]);
      }
      tc_fence_before();
      mbar_arrive(acc_free);
    }
    if (alive && i < L && (D > 32 || w == 0)) {
      float4* out = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dq) + ((size_t)bh * L + i) * D + C::W_OUT * w);
#pragma unroll
      for (int c = 0; c < C::W_OUT / 4; ++c)
        out[c] = make_float4(acc[4 * c] * scale, acc[4 * c + 1] * scale, acc[4 * c + 2] * scale, acc[4 * c + 3] * scale);
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

// The launch that owns keys: CTA = one 128-row key tile, thread <-> key row <-> TMEM lane; group w takes the queries
// [32 w, 32 w + 32) of a 64-query tile, and half of the columns of dK and dV in its registers.  lse and delta are per column here:
// warp 2 puts them into shared memory a tile ahead.
// Shared memory: the parts of K and V (D = 128: the lo part of K in TMEM), and the ring: Q and gO for the scores, gO and Q once more
// for dV and dK.  TMEM as in the forward: two score buffers [S | X = V gO^T], the parts of P over S and of gS over X, their lo
// parts beside them, one accumulator of 128 columns ([dV | dK], D = 128: dV, then dK).
// S has the forward's bits: its instructions come in the forward's order, for which all of a tile's Q stays in the ring until S is
// formed.  With the small products ordered by the parts of Q, as those of X are by the parts of gO, P was off by what S had lost to
// truncation in another way: dV of rows with one key 1.4e-6 from 64 bits at |S| of 50 (D = 128; 0 now), of dense rows 3.2e-6 (1.3e-6
// now, 2.3e-6 on the register-tiled kernels).  us of this launch, B2 H8 L1024, so / now: D128 155 / 141, D64 72 / 71, D32 61 / 64.
template <int D_>
struct DkvF32Cfg {
  static constexpr int D = D_;
  static constexpr int OWN = 128, BN = 64;
  static constexpr int NSL = D > 64 ? 2 : 1;
  static constexpr int KS = D < 64 ? D / 16 : 4;
  static constexpr int NTHREADS = 384;
  static constexpr bool KLO_TMEM = D > 64;
  static constexpr int K_PARTS = KLO_TMEM ? 2 : 3;
  static constexpr int PART = OWN * 128;
  static constexpr int TILE = BN * 128;
  static constexpr int OFF_V = K_PARTS * NSL * PART;
  static constexpr int OFF_RING = OFF_V + 3 * NSL * PART;
  static constexpr int STAT_BYTES = 2 * BN * 8;  // two tiles of (lse, delta)
  static constexpr int BUDGET = 227 * 1024 - 1024 - STAT_BYTES - 512;
  static constexpr int FIT = (BUDGET - OFF_RING) / TILE;
  static constexpr int STAGES = FIT > 16 ? 16 : FIT;
  static_assert(STAGES >= 3 * NSL + 2 && (STAGES & (STAGES - 1)) == 0, "a tile's Q stays until S is formed");
  static constexpr int OFF_STAT = OFF_RING + STAGES * TILE;
  static constexpr int OFF_BAR = OFF_STAT + STAT_BYTES;
  static constexpr int SMEM_NEEDED = OFF_BAR + 512 + 1024;
  static constexpr int SMEM_BYTES = SMEM_NEEDED > 120 * 1024 ? SMEM_NEEDED : 120 * 1024;  // one CTA per SM: it allocates all of TMEM
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static constexpr int SC = 128, COL_X = 64;
  static constexpr int COL_LO = 2 * SC;  // lo parts of P and gS
  static constexpr int COL_ACC = COL_LO + 64;
  static constexpr int COL_KLO = COL_ACC + 128;
  static constexpr int PIECES = NSL;
  static constexpr int W_OUT = 32 * NSL;  // columns of dK (and of dV) that a thread keeps
};

template <int D_, int MK>
__global__ void __launch_bounds__(384, 1)
bwd_f32_dkdv_kernel(const jvpfa_bwd_args a, const __grid_constant__ CUtensorMap map, const __nv_bfloat16* parts, int* status) {
  using C = DkvF32Cfg<D_>;
  constexpr int D = C::D, OWN = C::OWN, BN = C::BN, STAGES = C::STAGES, NSL = C::NSL, KS = C::KS;
  const bool dead_on_entry = *(volatile int*)(status + kF32GaveUp) != 0;

  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  float2* stats = reinterpret_cast<float2*>(smem + C::OFF_STAT);  // [2][BN]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* a_full = bars + 0;
  uint64_t* klo_full = bars + 1;   // 256
  uint64_t* s_full = bars + 2;     // [2]
  uint64_t* p_full = bars + 4;     // [2], 256
  uint64_t* acc_full = bars + 6;
  uint64_t* acc_free = bars + 7;   // 256
  uint64_t* stat_full = bars + 8;  // [2]
  uint64_t* full = bars + 10;      // [STAGES]
  uint64_t* empty = full + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + STAGES);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  const int BH = a.B * a.H;
  const int own0 = (int)blockIdx.x * OWN;  // (causal: the first key tile sees every query, and comes first)
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL;
  int n_valid = L;
  if (a.mask.kind == JVPFA_MASK_KVLEN) {
    const int n = a.mask.kv_len[b];
    n_valid = n < 0 ? 0 : (n > L ? L : n);
  }
  const int i_begin = causal ? own0 : 0;  // a multiple of BN
  const int n_tiles = own0 < n_valid ? (L - i_begin + BN - 1) / BN : 0;

  auto poison = [&]() {
    if (tid < OWN && own0 + tid < L) {
      poison_row<float>(a.dk, (size_t)bh * L + own0 + tid, D);
      poison_row<float>(a.dv, (size_t)bh * L + own0 + tid, D);
    }
  };
  if (dead_on_entry) {
    poison();
    return;
  }

  if (tid == 0) {
    mbar_init(a_full, 1);
    mbar_init(klo_full, 256);
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_full + s, 256);
      mbar_init(stat_full + s, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_free, 256);
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

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0 && n_tiles > 0) {
        prefetch_tmap(&map);
        auto load = [&](unsigned char* dst, uint64_t* bar, int slot, int part, int x, int y) {
          tma_load_4d(dst, &map, bar, x, y, bh, slot * 3 + part);
        };
        mbar_expect_tx(a_full, (C::K_PARTS + 3) * NSL * C::PART);
        for (int p = 0; p < 3; ++p)
          for (int s = 0; s < NSL; ++s)
            for (int r = 0; r < 2; ++r) {  // rows own0 + 64 r: beyond the tensor they read as zeros
              const int off = (p * NSL + s) * C::PART + r * C::TILE;
              if (p < C::K_PARTS) load(smem + off, a_full, kDqSlotK, p, 64 * s, own0 + 64 * r);
              load(smem + C::OFF_V + off, a_full, kDqSlotV, p, 64 * s, own0 + 64 * r);
            }
        int st = 0;
        uint32_t ph = 1;
        bool ok = true;
        auto unit = [&](int t, int slot, int p, int s) {
          if (!ok || !(ok = mbar_wait_backoff<64>(empty + st, ph, ab, kAbortBwdLoopEmpty))) return;
          mbar_expect_tx(full + st, C::TILE);
          load(smem + C::OFF_RING + st * C::TILE, full + st, slot, p, 64 * s, i_begin + t * BN);
          if (++st == STAGES) st = 0, ph ^= 1;
        };
        auto units = [&](int t, int slot) {  // one part and slice after another, the lo parts first
          for (int p = 2; p >= 0; --p)
            for (int s = 0; s < NSL; ++s) unit(t, slot, p, s);
        };
        auto scores = [&](int t) {
          for (int s = 0; s < NSL; ++s)
            for (int p = 0; p < 3; ++p) unit(t, kDqSlotQ, p, s);
          units(t, kDqSlotA);
        };
        scores(0);
        for (int t = 0; ok && t < n_tiles; ++t) {
          if (t + 1 < n_tiles) scores(t + 1);
          units(t, kDqSlotA), units(t, kDqSlotQ);
        }
      }
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer: a converged warp, one elected lane
      if (n_tiles > 0) {
        constexpr int F = Fmt<__nv_bfloat16>::kIdesc;
        constexpr uint32_t id64 = make_idesc(F, OWN, 64, 0, 0), id64t = make_idesc(F, OWN, 64, 0, 1);  // B K-major, MN-major
        constexpr uint32_t kLoMN = (uint32_t)(C::TILE >> 4) << 16;  // (one 64-column chunk: the leading offset is not used)
        constexpr uint32_t PART16 = C::PART >> 4, TILE16 = C::TILE >> 4;
        const uint32_t k_lo = kDescLo | (smem_u32(smem) >> 4), v_lo = kDescLo | (smem_u32(smem + C::OFF_V) >> 4);
        const uint32_t ring16 = smem_u32(smem + C::OFF_RING) >> 4;
        int st = 0;
        uint32_t ph = 0;
        bool ok = mbar_wait_warp(a_full, 0, ab, kAbortBwdOwn);
        if (C::KLO_TMEM && ok) ok = mbar_wait_warp(klo_full, 0, ab, kAbortBwdOwn);
        auto acquire = [&]() -> bool {
          if (!mbar_wait_warp(full + st, ph, ab, kAbortBwdLoopFull)) return ok = false;
          tc_fence_after();
          return true;
        };
        auto next = [&]() {
          if (++st == STAGES) st = 0, ph ^= 1;
        };
        auto stage = [&](int n) { return (st + n) & (STAGES - 1); };  // of the n-th unit from here
        auto scores = [&](int t) {
          const uint32_t sc = tmem + (t & 1) * C::SC;
          // S = K Q^T in the forward's order: parts lo, mid, hi of K, and beside each the small parts of Q first.  Unit 3 s + p from
          // here holds part p (hi, mid, lo) of slice s of Q; it is first used beside part 2 - p of K, and a slice's units are free
          // after its last product.
#pragma unroll
          for (int p = 2; p >= 0; --p) {
#pragma unroll
            for (int s = 0; s < NSL; ++s) {
              if (!mbar_wait_warp(full + stage(3 * s + 2 - p), ph ^ (st + 3 * s + 2 - p >= STAGES), ab, kAbortBwdLoopFull)) {
                ok = false;
                return;
              }
              tc_fence_after();
              if (elect_one()) {
#pragma unroll
                for (int pq = 2 - p; pq >= 0; --pq) {
                  const uint32_t bk = kDescLo | (ring16 + stage(3 * s + pq) * TILE16);
#pragma unroll
                  for (int ks = 0; ks < KS; ++ks) {
                    const uint32_t al = k_lo + (p * NSL + s) * PART16 + ks * 2;
                    const bool fresh = p == 2 && s == 0 && ks == 0;
                    if (C::KLO_TMEM && p == 2) {
                      if (fresh)
                        umma_ts_lo<false>(sc, tmem + C::COL_KLO, bk, id64);
                      else
                        umma_ts_lo<true>(sc, tmem + C::COL_KLO + s * 32 + ks * 8, bk + ks * 2, id64);
                    } else if (fresh) {
                      umma_ss_lo<false>(sc, al, bk, id64);
                    } else {
                      umma_ss_lo<true>(sc, al, bk + ks * 2, id64);
                    }
                  }
                }
                if (p == 0) {
#pragma unroll
                  for (int x = 0; x < 3; ++x) tc_commit(empty + stage(3 * s + x));
                }
              }
            }
          }
          st += 3 * NSL;
          if (st >= STAGES) st -= STAGES, ph ^= 1;
          // X = V gO^T
#pragma unroll
          for (int p = 2; p >= 0; --p) {
#pragma unroll
            for (int s = 0; s < NSL; ++s) {
              if (!acquire()) return;
              const uint32_t bk = kDescLo | (ring16 + st * TILE16);
              if (elect_one()) {
#pragma unroll
                for (int pa = 2 - p; pa >= 0; --pa) {  // small products first
#pragma unroll
                  for (int ks = 0; ks < KS; ++ks) {
                    if (p == 2 && s == 0 && ks == 0)
                      umma_ss_lo<false>(sc + C::COL_X, v_lo, bk, id64);
                    else
                      umma_ss_lo<true>(sc + C::COL_X, v_lo + (pa * NSL + s) * PART16 + ks * 2, bk + ks * 2, id64);
                  }
                }
                tc_commit(empty + st);
                if (p == 0 && s == NSL - 1) tc_commit(s_full + (t & 1));
              }
              next();
            }
          }
        };
        int piece = 0;
        auto begin_piece = [&]() -> bool {
          if (piece > 0 && !mbar_wait_warp(acc_free, (piece - 1) & 1, ab, kAbortBwdDone)) return ok = false;
          tc_fence_after();
          ++piece;
          return true;
        };
        auto outputs = [&](int t) {
          const uint32_t sc = tmem + (t & 1) * C::SC;
          if (!mbar_wait_warp(p_full + (t & 1), (t >> 1) & 1, ab, kAbortBwdPFull)) {
            ok = false;
            return;
          }
#pragma unroll
          for (int side = 0; side < 2; ++side) {  // dV += P^T gO, dK += gS^T Q
            if (side < C::PIECES && !begin_piece()) return;
#pragma unroll
            for (int p = 2; p >= 0; --p) {
#pragma unroll
              for (int s = 0; s < NSL; ++s) {
                if (!acquire()) return;
                const uint32_t bm = kLoMN | (ring16 + st * TILE16);
                if (elect_one()) {
                  const uint32_t acc = tmem + C::COL_ACC + 64 * (NSL == 1 ? side : s);
#pragma unroll
                  for (int pa = 2 - p; pa >= 0; --pa) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {  // 16 queries
                      const uint32_t acol = pa < 2 ? sc + side * C::COL_X + 8 * pa + 16 * kk
                                                   : tmem + C::COL_LO + 32 * (kk >> 1) + 16 * side + 8 * (kk & 1);
                      if (p == 2 && kk == 0)
                        umma_ts_lo<false>(acc, acol, bm, id64t);
                      else
                        umma_ts_lo<true>(acc, acol, bm + kk * 128, id64t);
                    }
                  }
                  tc_commit(empty + st);
                  if (p == 0 && s == NSL - 1 && (side == 1 || C::PIECES == 2)) tc_commit(acc_full);
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
    } else if (warp == 2) {
      // ------------------------------------------------------------------ statistics of the queries
      for (int t = 0; t < n_tiles; ++t) {
        // (tile t - 2 has been read from this half; its phase cannot be followed by another before this tile's statistics are there)
        if (t >= 2 && !mbar_wait(p_full + (t & 1), ((t >> 1) - 1) & 1, ab, kAbortBwdPFull)) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = i_begin + t * BN + 32 * e + lane;
          const size_t at = (size_t)bh * L + min(i, L - 1);
          stats[(t & 1) * BN + 32 * e + lane] = i < L ? make_float2(a.lse[at], a.delta[at]) : make_float2(INFINITY, 0.f);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(stat_full + (t & 1));
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // ------------------------------------------------------------------ elementwise, dK and dV
    const int w = (warp - 4) >> 2;
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int j = own0 + row;  // key
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const float scale_log2 = a.sm_scale * kLog2e;
    if constexpr (C::KLO_TMEM) {
      // the lo part of this row of K, columns [64 w, 64 w + 64), to its 32 TMEM columns
      uint32_t r[32];
      const uint4* src = reinterpret_cast<const uint4*>(
          parts + ((size_t)(kDqSlotK * 3 + 2) * BH + bh) * L * D + (size_t)min(j, L - 1) * D + 64 * w);
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint4 v = j < L ? ldg_nc_v4(src + x) : make_uint4(0u, 0u, 0u, 0u);
        r[4 * x] = v.x, r[4 * x + 1] = v.y, r[4 * x + 2] = v.z, r[4 * x + 3] = v.w;
      }
      tmem_st32(tmem + lane_off + C::COL_KLO + 32 * w, r);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(klo_full);
    }
    const MaskView mv = make_mask_view(a.mask, b, h, L);
    const long long jo = (long long)min(j, L - 1) * mv.sj;
    float acc_k[C::W_OUT], acc_v[C::W_OUT];
#pragma unroll
    for (int x = 0; x < C::W_OUT; ++x) acc_k[x] = acc_v[x] = 0.f;
    int piece = 0;
    bool alive = true;
    // What the mask holds for a tile's queries (neighbouring lanes read neighbouring keys), requested a tile ahead as in the forward.
    float bias[MK == 2 ? 32 : 1];
    uint32_t next_live = 0u;
    auto fetch_mask = [&](int t) {
      const int i0 = i_begin + min(t, n_tiles - 1) * BN + 32 * w;
      next_live = j < n_valid ? first_columns(L - i0) : 0u;  // queries that attend this key, a bit each
      if (causal) next_live &= ~first_columns(j - i0);
      if constexpr (MK == 1) {
        uint32_t r = 0u;
#pragma unroll 8
        for (int c = 0; c < 32; ++c)
          r |= (ldg_nc_u8(reinterpret_cast<const unsigned char*>(mv.base) + (long long)min(i0 + c, L - 1) * mv.si + jo) != 0u ? 1u : 0u) << c;
        next_live &= r;
      }
      if constexpr (MK == 2) {
#pragma unroll
        for (int c = 0; c < 32; ++c) bias[c] = mv.bias(min(i0 + c, L - 1), min(j, L - 1));
      }
    };
    if (n_tiles > 0) fetch_mask(0);
    for (int t = 0; alive && t < n_tiles; ++t) {
      const uint32_t tS = tmem + lane_off + (t & 1) * C::SC + 32 * w, tLO = tmem + lane_off + C::COL_LO + 32 * w;
      const uint32_t live = next_live;
      if (!mbar_wait(stat_full + (t & 1), (t >> 1) & 1, ab, kAbortBwdLoopFull) ||
          !mbar_wait(s_full + (t & 1), (t >> 1) & 1, ab, kAbortBwdSFull)) {
        alive = false;
        break;
      }
      tc_fence_after();
      const float4* st = reinterpret_cast<const float4*>(stats + (t & 1) * BN + 32 * w);
#pragma unroll
      for (int s = 0; s < 2; ++s) {  // 16 queries at a time: one contraction step of the output products
        uint32_t x[16], y[16];
        tmem_ld16(tS + 16 * s, x);
        tmem_ld16(tS + C::COL_X + 16 * s, y);
        tmem_wait_ld();
        uint32_t ph[16], pl[8];  // hi parts, then mid parts ; lo parts
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 q2 = st[8 * s + c];  // lse, delta of two queries
          float p[2], g[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int n = 2 * c + e;
            const float v = f32_score<MK>(__uint_as_float(x[n]), scale_log2, MK == 2 ? bias[16 * s + n] : 0.f);
            const bool ok = (live >> (16 * s + n)) & 1u;  // (nothing of a masked pair counts, whatever it is)
            p[e] = ok ? fast_exp2(v - (e ? q2.z : q2.x)) : 0.f;
            g[e] = ok ? p[e] * (__uint_as_float(y[n]) - (e ? q2.w : q2.y)) : 0.f;
          }
          split3_pair(p[0], p[1], ph[c], ph[8 + c], pl[c]);
          y[2 * c] = __float_as_uint(g[0]), y[2 * c + 1] = __float_as_uint(g[1]);
        }
        tmem_st16(tS + 16 * s, ph);
        tmem_st8(tLO + 8 * s, pl);
#pragma unroll
        for (int c = 0; c < 8; ++c) split3_pair(__uint_as_float(y[2 * c]), __uint_as_float(y[2 * c + 1]), ph[c], ph[8 + c], pl[c]);
        tmem_st16(tS + C::COL_X + 16 * s, ph);
        tmem_st8(tLO + 16 + 8 * s, pl);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(p_full + (t & 1));
      fetch_mask(t + 1);
#pragma unroll
      for (int pc = 0; pc < C::PIECES; ++pc) {
        if (!mbar_wait(acc_full, piece & 1, ab, kAbortBwdDone)) {
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
          for (int c = 0; c < 32; ++c) acc[c] += __uint_as_float(r[c]);
        };
        if constexpr (NSL == 1) {
          add(acc_v, tA + 32 * w);
          add(acc_k, tA + 64 + 32 * w);
        } else if (pc == 0) {
          add(acc_v, tA + 64 * w);
          add(acc_v + 32, tA + 64 * w + 32);
        } else {
          add(acc_k, tA + 64 * w);
          add(acc_k + 32, tA + 64 * w + 32);
        }
        tc_fence_before();
        mbar_arrive(acc_free);
      }
    }
    if (alive && j < L && (D > 32 || w == 0)) {
      const size_t at = ((size_t)bh * L + j) * D + C::W_OUT * w;
      float4* pk = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dk) + at);
      float4* pv = reinterpret_cast<float4*>(reinterpret_cast<float*>(a.dv) + at);
      const float scale = a.sm_scale;
#pragma unroll
      for (int c = 0; c < C::W_OUT / 4; ++c) {
        pk[c] = make_float4(acc_k[4 * c] * scale, acc_k[4 * c + 1] * scale, acc_k[4 * c + 2] * scale, acc_k[4 * c + 3] * scale);
        pv[c] = make_float4(acc_v[4 * c], acc_v[4 * c + 1], acc_v[4 * c + 2], acc_v[4 * c + 3]);
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

template <typename C>
static int launch_bwd_f32_kernel(void (*kern)(jvpfa_bwd_args, CUtensorMap, const __nv_bfloat16*, int*), SmemOptIn& opt_in,
                                 const jvpfa_bwd_args& a, const CUtensorMap& map, int* status, cudaStream_t stream) {
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return JVPFA_ERR_CUDA;
  const dim3 grid((a.L + 127) / 128, a.B * a.H);
  kern<<<grid, C::NTHREADS, C::SMEM_BYTES, stream>>>(a, map, static_cast<const __nv_bfloat16*>(a.workspace), status);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch bwd_f32_tc5");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <int D, int MK>
static int launch_bwd_f32_mk(const jvpfa_bwd_args& a, const CUtensorMap& map, int* status, cudaStream_t s) {
  static SmemOptIn opt_kv, opt_o, opt_t;
  int rc = JVPFA_OK;
  if (!(a.flags & JVPFA_SKIP_DKDV)) rc = launch_bwd_f32_kernel<DkvF32Cfg<D>>(bwd_f32_dkdv_kernel<D, MK>, opt_kv, a, map, status, s);
  if (rc || (a.flags & JVPFA_SKIP_DQ)) return rc;
  if (a.gto) return launch_bwd_f32_kernel<DqF32Cfg<D, true>>(bwd_f32_dq_kernel<D, true, MK>, opt_t, a, map, status, s);
  return launch_bwd_f32_kernel<DqF32Cfg<D, false>>(bwd_f32_dq_kernel<D, false, MK>, opt_o, a, map, status, s);
}

template <int D>
static int launch_bwd_f32_d(const jvpfa_bwd_args& a, const CUtensorMap& map, int* status, cudaStream_t s) {
  if (a.mask.kind == JVPFA_MASK_BOOL) return launch_bwd_f32_mk<D, 1>(a, map, status, s);
  if (a.mask.kind == JVPFA_MASK_BIAS) return launch_bwd_f32_mk<D, 2>(a, map, status, s);
  return launch_bwd_f32_mk<D, 0>(a, map, status, s);
}

}  // namespace tc5

long long bwd_f32_tc5_workspace(const jvpfa_bwd_args& a) {
  if (a.dtype != JVPFA_FP32 || a.impl == JVPFA_IMPL_GENERIC) return 0;
  if (a.gto && (a.go || !(a.flags & JVPFA_ZERO_TKV) || !(a.flags & JVPFA_SKIP_DKDV))) return 0;
  if (a.impl == JVPFA_IMPL_AUTO && !tc5::f32_rows_enough(a.mask, a.B, a.H, a.L, a.D)) return 0;
  return (long long)(a.gto ? 5 : 4) * 3 * 2 * a.B * a.H * a.L * a.D;
}

bool bwd_f32_tc5_eligible(const jvpfa_bwd_args& a) {
  const long long need = bwd_f32_tc5_workspace(a);
  return need > 0 && a.workspace != nullptr && a.workspace_bytes >= need && (reinterpret_cast<uintptr_t>(a.workspace) & 15u) == 0;
}

int launch_bwd_f32_tc5(const jvpfa_bwd_args& a, cudaStream_t stream) {
  using namespace tc5;
  int* status = tc5_status_device_ptr();
  if (!status) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  const int slots = a.gto ? 5 : 4;
  SplitArgs s{};
  s.dst = static_cast<__nv_bfloat16*>(a.workspace);
  s.plane = (long long)a.B * a.H * a.L * a.D;
  s.H = a.H, s.L = a.L, s.D = a.D;
  if (a.mask.kind == JVPFA_MASK_KVLEN) s.kv_len = a.mask.kv_len, s.padded = 1u << kDqSlotK | 1u << kDqSlotV;
  // (dQ alone: the rows that attend such a key have a delta, or a cterm, that is not a number)
  if (a.mask.kind == JVPFA_MASK_CAUSAL && (a.flags & JVPFA_SKIP_DKDV)) s.clean = 1u << kDqSlotK | 1u << kDqSlotV;
  s.set(kDqSlotQ, a.q, a.in_stride), s.set(kDqSlotK, a.k, a.in_stride), s.set(kDqSlotV, a.v, a.in_stride);
  if (a.gto) {
    s.set(kDqSlotA, a.tq, a.in_stride), s.set(kDqSlotB, a.gto, nullptr);
  } else {
    s.set(kDqSlotA, a.go, nullptr);
  }
  CUtensorMap map;
  if (!encode_map_parts(&map, a.workspace, a.D, a.L, a.B * a.H, slots * 3)) {
    set_last_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled(bwd f32)");
    return JVPFA_ERR_CUDA;
  }
  const int rc = launch_split3(s, slots, stream);
  if (rc) return rc;
  if (a.D == 32) return launch_bwd_f32_d<32>(a, map, status, stream);
  if (a.D == 64) return launch_bwd_f32_d<64>(a, map, status, stream);
  return launch_bwd_f32_d<128>(a, map, status, stream);
}

}  // namespace jvpfa
