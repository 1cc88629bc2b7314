// Single-pass tcgen05 backward for head dimension 64 (bf16 / fp16): the score
// tiles S, tS, E, FP are formed ONCE per (128 keys x 64 queries) sub-tile and feed all three gradients.
//
// The two-launch backward (bwd_tc5_d64.cu, like upstream's _attn_bwd_dkdv / _attn_bwd_dq,
// jvp_attention.py:1415-1707) recomputes the score tiles in the launch that owns queries: 15 MMAs are
// executed for 10 needed.  Here one persistent CTA per SM owns 128 keys (keys <-> TMEM lanes), streams the
// queries in sub-tiles of 64 and produces
//     dK += gS^T Q + gtS^T tQ,   dV += A^T G (+ P^T gO)            accumulated in TMEM over the sub-tiles,
//     dQ[sub-tile] = gS K + gtS tK                                 one 64 x 64 product per sub-tile,
// The dQ product contracts over the keys, i.e. over TMEM lanes, so its operands cannot come from TMEM: the
// elementwise threads write gS and gtS as 16-bit tiles [key][query] into SHARED memory.  That one layout is a
// K-major A operand for the dK products (M = keys) and an MN-major A operand for the dQ product (M = 64
// queries, K = keys); K / tK are its MN-major B operand.  A and P, which only dV needs, stay in TMEM.  Handing the operands over through
// shared memory also frees the score accumulators as soon as the elementwise threads hold them in
// registers, so the scores of sub-tile g+1 are formed while sub-tile g is still being worked on.
// A dQ sub-tile is read back by a fourth warpgroup (an M = 64 accumulator sits in lanes 0..15 of each
// 32-lane quarter) and added to an fp32 accumulation buffer in global memory with TMA reductions; a small kernel converts that
// buffer to the output type at the end.  The order of those additions varies from run to run, so dQ is reproducible to
// rounding, not bitwise.  (With a bias and through tO a key tile's share is stored instead, see dq_parts; at D = 32 always.)
//
// Measured on a B200, cycles of a sub-tile inside an item (clock marks in one CTA, every SM at work): through O 1660, through tO 2310,
// both 2600; the tensor pipe's own time is 1024, 1860 and 2050, so that with tangents it is busy four fifths of a sub-tile, and
// through O the elementwise threads are (two warps for a scheduler, so their latencies show).  A key tile's beginning costs 7.6 k
// cycles more.  Before the looks at the barriers were taken together and dV's products went first: 2060, 2760, 3130.
//
// Warps: 0 TMA producer (+ per-query statistics), 1 score issuer, 2 dK/dV issuer, 3 dQ issuer,
// 4..11 two elementwise warpgroups (thread <-> key row; group w takes query columns [32w, 32w+32) of every
// sub-tile), 12..15 dQ read-back.  (Four elementwise warpgroups of 16 columns each, taking turns at the
// read-back, were measured slower: 0.284 ms against 0.261 ms on the B4 H16 L2048 causal shape.)
// TMEM (512 columns): S | tS | E | FP (64 each) ; dK | dV (64 each) ; dQ (64) ; packed A | P (32 each).
#include "tc5_common.cuh"

namespace jvpfa {
namespace tc5 {

struct BwdFMaps {
  CUtensorMap k, v, tk, tv;  // key side, box 128 rows
  CUtensorMap q, go, tq, g;  // query side, box 64 rows (g = cotangent of tO)
  CUtensorMap dq;            // the fp32 dQ accumulation buffer, box 64 rows x 32 columns
};

// TMA reduction (add) of one fp32 tile from shared memory into global memory; rows past the tensor's extent are
// not touched.
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, uint32_t smem_src, int x, int y, int z, int w) {
  asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
               "r"(smem_src), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
// The same as a plain store.
__device__ __forceinline__ void tma_store_part_4d(const CUtensorMap* map, uint32_t smem_src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(smem_src),
               "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <bool HAS_GO, bool HAS_GT>
struct BwdFCfg {
  static constexpr int D = 64;
  static constexpr int OWN = 128;
  static constexpr int BL = 64;
  // The streamed tiles go through one ring, or, where three stages of all four would not fit, through two: Q and tQ three
  // stages deep, G and gO two.  With two stages of everything the scores of sub-tile g + 2 waited for the outputs of g and then
  // for the loads (half of the score issuer's time).
  static constexpr bool TWO_RINGS = HAS_GO && HAS_GT;
  static constexpr int STAGES = 3;
  static constexpr int GSTAGES = TWO_RINGS ? 2 : STAGES;  // (also the stages of the statistics)
  // The shared-memory result tiles (gS, gtS) exist twice, so that the elementwise threads can write sub-tile g + 1
  // while the products of sub-tile g still read theirs.
  static constexpr int N_OBUF = 2;
  static constexpr int NTHREADS = 512;
  static constexpr int N_OWN = HAS_GT ? 4 : 2;                           // K, tK, V, tV | K, V
  static constexpr int N_LOOP = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0);  // Q, tQ, G, gO
  static constexpr int N_OUT = 1 + (HAS_GT ? 1 : 0);                      // gS, gtS (A and P stay in TMEM)
  static constexpr int OWN_BYTES = OWN * D * 2;   // 16 KiB
  static constexpr int LOOP_BYTES = BL * D * 2;   // 8 KiB
  static constexpr int OUT_BYTES = OWN * BL * 2;  // 16 KiB: [128 keys][64 queries]
  static constexpr int STAGE_BYTES = (TWO_RINGS ? 2 : N_LOOP) * LOOP_BYTES;
  static constexpr int G_STAGE_BYTES = TWO_RINGS ? 2 * LOOP_BYTES : 0;
  static constexpr int STAT_STAGE_BYTES = (BL / 2) * 32;  // per query pair two float4
  // Two sets of own tiles where shared memory allows it (backward through O alone: K and V only): the next item's
  // are then loaded while this item's last sub-tiles run.  With one set the item boundary is exposed - the next
  // load can only be requested when the last dQ product has completed (about an eighth of the kernel's time).
  static constexpr int OWN_BUFS = HAS_GT ? 1 : 2;
  static constexpr int OWN_SET_BYTES = N_OWN * OWN_BYTES;
  static constexpr int OFF_OWN = 0;
  static constexpr int OFF_RING = OWN_BUFS * OWN_SET_BYTES;
  static constexpr int OFF_GRING = OFF_RING + STAGES * STAGE_BYTES;
  static constexpr int OFF_OUT = OFF_GRING + GSTAGES * G_STAGE_BYTES;
  static constexpr int OBUF_BYTES = N_OUT * OUT_BYTES;
  static constexpr int OFF_STAT = OFF_OUT + N_OBUF * OBUF_BYTES;
  // dQ of a sub-tile on its way out: fp32 [64 queries][64 columns] as two 128-byte-swizzled halves of 32 columns
  static constexpr int OFF_DQS = OFF_STAT + GSTAGES * STAT_STAGE_BYTES;
  static constexpr int DQS_BYTES = BL * D * 4;
  static_assert(OFF_DQS % 1024 == 0, "swizzled staging tile alignment");
  static constexpr int TILE_BYTES = OFF_DQS + DQS_BYTES;
  static constexpr int SMEM_NEEDED = TILE_BYTES + 512;
  // At least 120 KiB so that a second CTA can never share the SM (the CTA allocates all of TMEM).
  static constexpr int SMEM_BYTES = SMEM_NEEDED > 120 * 1024 ? SMEM_NEEDED : 120 * 1024;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static constexpr int SLOT_K = 0, SLOT_TK = 1, SLOT_V = HAS_GT ? 2 : 1, SLOT_TV = 3;
  static constexpr int SLOT_Q = 0, SLOT_TQ = 1, SLOT_G = TWO_RINGS ? 0 : 2, SLOT_GO = HAS_GT ? SLOT_G + 1 : 1;
  static constexpr int OUT_GS = 0, OUT_GT = 1;
  static constexpr int COL_S = 0, COL_TS = 64, COL_E = 128, COL_FP = HAS_GT ? 192 : 64;
  static constexpr int COL_DK = 256, COL_DV = 320, COL_DQ = 384;
  static constexpr int COL_AV = 448, COL_P = 480;  // packed 16-bit A and P: TMEM operands of the dV products
  static constexpr int COLS_ALLOC = 512;
};

__device__ __forceinline__ float2 ff(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ void sts_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// D[tmem] (+)= A[smem] * B[smem]; descriptor low words as in umma_ss_lo, accumulate flag known at run time.
__device__ __forceinline__ void mma_ss_dyn(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}

struct FItem {
  int bh, b, h, own0, loop_begin, n_sub;  // a key tile and the n_sub sub-tiles of it that are this CTA's
};

// ---- Key tiles shared out among CTAs -----------------------------------------------------------
// Dealt whole, 192 key tiles take two rounds of 148 CTAs where 1.3 rounds' worth of work is there, and 32 key tiles leave 116 SMs idle.
// With a workspace the sub-tiles of all key tiles are one line that is cut into as many equal pieces as there are CTAs; a key
// tile that is cut leaves its shares of dK and dV (fp32) in the workspace, and the kernel that converts dQ adds them up in their
// order.  The line is ordered by head, key tile, sub-tile; a key tile's beginning (own tiles, first scores, epilogue) counts as kOpen
// sub-tiles.  Measured on a B200 (start of the kernel, a sub-tile, a beginning; us): through O 5, 0.9, 2; through tO 7, 1.4, 2; both 6,
// 1.7, 3.
//
// Dealt whole -> shared out, us with the kernel that follows, bf16, H24 L1024 / H4 L1024: through O 41.9 -> 35.9 / 21.6 -> 16.0, through tO
// 59.6 -> 51.0 / 29.2 -> 20.2, both 70.4 -> 58.8 / 34.5 -> 22.0; B2 H12 L2048 with a boolean mask through tO 169 -> 158; fp16 B8 H12 L1024,
// lengths in [L/2, L], both 177 -> 155.
constexpr int kOpen = 2;
constexpr int kShareFloats = 128 * 64;             // one share of dK or dV, in 16-byte pieces: [16 pieces][128 keys]
constexpr long long kShareHead = 16 * 1024;        // bytes: where each CTA begins, {key tile, sub-tile}
constexpr long long split_bytes(int ctas) { return kShareHead + (long long)ctas * 4 * kShareFloats * 4; }

__device__ __forceinline__ int2 split_begin(const jvpfa_bwd_args& a, int c, int G) {
  const int slope = a.mask.kind == JVPFA_MASK_CAUSAL ? -2 : 0, first = (a.L + 63) / 64;
  return cut_begin(
      a.mask.kind == JVPFA_MASK_KVLEN, a.B, a.H, (a.L + 127) / 128, slope, kOpen, 0, c, G,
      [&](int b) { return ((a.mask.kind == JVPFA_MASK_KVLEN ? max(0, min(a.mask.kv_len[b], a.L)) : a.L) + 127) / 128; },
      [&](int) { return first; }, [&](int, int r) { return first + slope * r; });
}

// MK: 0 = none / causal / key padding (index comparisons); 1 = boolean mask, as bits or as bytes of any strides (each elementwise
// thread requests the next sub-tile's 32 entries of its key when the scores of this one have left its registers); 2 = additive
// bias of the element type, requested the same way.
//
// dQ of a bias call through tO is summed in a fixed order, as the two launches that served it sum it: a key tile's share goes to
// a buffer of its own (dq_acc: [key tile][B*H][L][D] floats) and fused64_finish_kernel adds them up.  Measured on a B200, the two
// launches / this with the sum, us, bf16 through both outputs: B2 H12 L512 34 / 25, L1024 121 / 75, L2048 342 / 255, H4 L4096
// 226 / 172; with 48 key tiles (B2 H12 L256) 22 / 28, with 32 (H1 L4096) 124 / 173, both before key tiles were shared out.
//
// At head dimension 32 it always is, whatever the mask and the cotangents (key padding and tile bitmaps keep the two launches): tensor maps end at
// column 32, contractions over D stop half-way, and a key tile's share of dQ has half the bytes.  Two launches / this with the sum, us, bf16 through
// O / tO / both: B4 H8 L1000 56 / 40, 70 / 54, 78 / 58; B1 H5 L4096 177 / 83, 225 / 112, 254 / 124; B5 H9 L1732 with a bias 649 / 318, 723 / 384,
// 736 / 424; B4 H16 L2048 causal 173 / 137, 221 / 195, 249 / 222; B8 H12 L130 21 / 16, 24 / 20, 25 / 21; B1 H1 L1024 20 / 14, 24 / 17, 26 / 18.
__host__ __device__ __forceinline__ bool dq_parts(const jvpfa_bwd_args& a) {
  return a.D == 32 || (a.mask.kind == JVPFA_MASK_BIAS && a.gto != nullptr);
}
// HD: the head dimension, 64 or 32.  RAG, of a bias: its length is not a multiple of 16.  (Known at run time alone they cost the D = 64 kernels up to
// 4 and 5 %.)
template <typename T, bool HAS_GO, bool HAS_GT, int MK, bool CUT, int HD, bool RAG>
__global__ void __launch_bounds__(512, 1)
bwd_tc5_fused64_kernel(const jvpfa_bwd_args a, const __grid_constant__ BwdFMaps maps, float* dq_acc, float* shares, int* status) {
  using C = BwdFCfg<HAS_GO, HAS_GT>;
  constexpr int D = 64, OWN = C::OWN, BL = C::BL, STAGES = C::STAGES, GSTAGES = C::GSTAGES;

  behind_previous();
  const bool dead_on_entry = *(volatile int*)status != 0;  // an earlier bounded wait gave up

  extern __shared__ __align__(1024) unsigned char smem[];  // (the tiles' swizzle repeats every 1024 bytes)
  unsigned char* sOwn = smem + C::OFF_OWN;
  unsigned char* sRing = smem + C::OFF_RING;
  unsigned char* sOut = smem + C::OFF_OUT;
  unsigned char* sG = smem + C::OFF_GRING;
  float4* sStat = reinterpret_cast<float4*>(smem + C::OFF_STAT);  // [GSTAGES][BL/2][2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::TILE_BYTES);
  uint64_t* own_full = bars + 0;             // [2] per set of own tiles (item kact uses set kact % OWN_BUFS)
  uint64_t* own_free = bars + 2;             // [2] score issuer + dQ issuer are through with the set
  uint64_t* loop_full = bars + 4;            // [STAGES]
  uint64_t* loop_empty = loop_full + STAGES;  // [STAGES]: score issuer + dK/dV issuer
  uint64_t* g_full = loop_empty + STAGES;     // [2] TWO_RINGS: the same of G and gO
  uint64_t* g_empty = g_full + 2;             // [2]
  uint64_t* stat_full = g_empty + 2;          // [GSTAGES]
  uint64_t* s_full = stat_full + GSTAGES;
  uint64_t* s_free = s_full + 1;    // 256 elementwise threads hold the scores in registers
  // [2] by g & 1, 256 each: gS, gtS, A, P of the sub-tile are in shared memory. A pair, because the elementwise
  // threads can finish sub-tile g + 1 before the dQ issuer has looked at g (sub-tile g + 1 needs the dV products of
  // g, not its dQ product): on one barrier the issuer would then be two phases behind, where a parity wait no longer
  // tells "done" from "not yet". Sub-tile g + 2 does need dQ of g (out_free), so one phase per barrier is the most.
  uint64_t* p_full = s_free + 1;
  uint64_t* out_free = p_full + 2;  // [2] per result buffer: dK/dV issuer + dQ issuer have read it
  uint64_t* av_free = out_free + 2;  // the dV products have read the packed A / P columns
  uint64_t* dq_full = av_free + 1;
  uint64_t* dq_free = dq_full + 1;   // 128 read-back threads
  uint64_t* done = dq_free + 1;      // the item's dK / dV are complete
  uint64_t* acc_free = done + 1;     // 256: the epilogue has read them
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* rb_ok = reinterpret_cast<volatile int*>(tmem_slot + 2);  // the read-back group's poller tells the rest

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int L = a.L;
  const int BH = a.B * a.H;
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL;
  const int n_own_tiles = (L + OWN - 1) / OWN;
  const int n_items = n_own_tiles * BH;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  unsigned char* order = smem + C::TILE_BYTES + 256;  // behind the barriers
  int* s_cut = reinterpret_cast<int*>(smem + C::TILE_BYTES + 384);  // CUT: {key tile, sub-tile} where this CTA and the next begin
  const bool sorted = !CUT && a.mask.kind == JVPFA_MASK_KVLEN && a.B <= kMaxSortedBatch && n_items > G;
  if constexpr (CUT) {
    if (warp < 2) {
      const int2 at = split_begin(a, cta + warp, G);
      if (lane == 0) {
        s_cut[2 * warp] = at.x, s_cut[2 * warp + 1] = at.y;
        if (warp == 0) reinterpret_cast<int2*>(shares)[cta] = at;
      }
    }
    __syncthreads();
  } else if (sorted) {
    sort_batch(a.mask, a.B, order);
    __syncthreads();
  }

  // This CTA's items, by `walk`: shared out, the key tile's number; dealt whole, the round, in serpentine order and ranked heaviest
  // first (causal: the first key tile sees every query).
  auto begin_items = [&]() { return CUT ? s_cut[0] : 0; };
  auto first_sub = [&](int w) { return w == s_cut[0] ? s_cut[1] : 0; };
  auto get_item = [&](int walk, FItem& it) -> bool {
    int rank, s0 = 0;
    if constexpr (CUT) {
      s0 = first_sub(walk);
      if (walk > s_cut[2] || (walk == s_cut[2] && s0 >= s_cut[3])) return false;
      it.bh = walk / n_own_tiles;
      rank = walk - it.bh * n_own_tiles;
    } else {
      const int w = walk * G + ((walk & 1) ? (G - 1 - cta) : cta);
      if (w >= n_items) return false;
      rank = w / BH;
      it.bh = w - rank * BH;
    }
    it.b = it.bh / a.H;
    it.h = it.bh - it.b * a.H;
    if (sorted) it.b = order[it.b], it.bh = it.b * a.H + it.h;
    int n_valid = L;
    if (a.mask.kind == JVPFA_MASK_KVLEN) {
      const int n = a.mask.kv_len[it.b];
      n_valid = n < 0 ? 0 : (n > L ? L : n);
    }
    it.own0 = rank * OWN;
    it.loop_begin = causal ? (it.own0 / BL) * BL : 0;
    it.n_sub = (L - it.loop_begin + BL - 1) / BL;
    if (it.own0 >= n_valid) it.n_sub = 0;
    if constexpr (CUT) {
      it.loop_begin += s0 * BL;
      it.n_sub = (walk == s_cut[2] ? s_cut[3] : it.n_sub) - s0;
    }
    return true;
  };
  // Place of an item's share, which = 0 dK, 1 dV; nullptr: the item is a whole key tile.
  auto share = [&](int walk, int which) -> float* {
    if (!CUT) return nullptr;
    const int place = cut_place(s_cut, walk, cta);
    return place < 0 ? nullptr : shares + kShareHead / 4 + (size_t)(2 * place + which) * kShareFloats;
  };
  auto valid_keys = [&](int b) {
    int n_valid = L;
    if (a.mask.kind == JVPFA_MASK_KVLEN) {
      const int n = a.mask.kv_len[b];
      n_valid = n < 0 ? 0 : (n > L ? L : n);
    }
    return n_valid;
  };

  constexpr bool parts = HD == 32 || (HAS_GT && MK == 2);  // dq_parts
  // NaN into the rows of dK, dV and of the dQ accumulator that this CTA's items own: this launch's results are
  // not to be trusted
  auto poison = [&]() {
    FItem it;
    for (int walk = begin_items(); get_item(walk, it); ++walk) {
      const int i = it.own0 + tid;
      if (tid < OWN && share(walk, 0)) share(walk, 0)[4 * tid] = share(walk, 1)[4 * tid] = poison_f32();
      if (tid < OWN && i < L) {
        poison_row<T>(a.dk, (size_t)it.bh * L + i, HD);
        poison_row<T>(a.dv, (size_t)it.bh * L + i, HD);
        dq_acc[((parts ? (size_t)(it.own0 / OWN) * BH * L : 0) + (size_t)it.bh * L + i) * HD] = poison_f32();
      }
    }
  };
  if ((smem_u32(smem) & 1023u) != 0) {  // (does not happen: the array is declared so)
    if (tid == 0) publish_abort(status, kAbortAux);
    poison();
    return;
  }
  if (dead_on_entry) {
    poison();
    return;
  }

  if (tid == 0) {
    mbar_init(own_full, 1);
    mbar_init(own_full + 1, 1);
    mbar_init(own_free, 2);
    mbar_init(own_free + 1, 2);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(loop_full + s, 1);
      mbar_init(loop_empty + s, 2);
      if (s < 2) mbar_init(g_full + s, 1), mbar_init(g_empty + s, 2);
      if (s < GSTAGES) mbar_init(stat_full + s, 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_free, 256);
    mbar_init(p_full, 256);
    mbar_init(p_full + 1, 256);
    mbar_init(out_free, 2);
    mbar_init(out_free + 1, 2);
    mbar_init(av_free, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 128);
    mbar_init(done, 1);
    mbar_init(acc_free, 256);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, C::COLS_ALLOC);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const AbortState ab{abort_flag, status};

  // Registers: the elementwise threads hold four 32-column accumulator slices; everybody else needs few.
  // (setmaxnreg.inc draws on what setmaxnreg.dec of the same CTA has released and blocks until it is there: 256
  // threads x 48 registers up equal 128 x 64 and 128 x 32 down from the 128 the kernel is launched with.  The read-back threads
  // hold 64 of a row and spilled at 72 and at 80: through tO at B4 H16 L2048 causal 204 and 195 us against 192.)
  // (It stands in the branches of the roles: ptxas holds code behind a join of the two to the smaller number.)
  // Phase counters kept alike by all roles: g counts the sub-tiles of this CTA (ring stage g % STAGES, dQ buffer
  // g & 1; s_full, s_free complete once per sub-tile, p_full and out_free of buffer g & 1 every other one), kact the items that have sub-tiles.
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer + per-query statistics
      if (lane == 0) {
        prefetch_tmap(&maps.k), prefetch_tmap(&maps.v), prefetch_tmap(&maps.q);
        if constexpr (HAS_GO) prefetch_tmap(&maps.go);
        if constexpr (HAS_GT) prefetch_tmap(&maps.tk), prefetch_tmap(&maps.tv), prefetch_tmap(&maps.tq), prefetch_tmap(&maps.g);
      }
      struct Stat {
        float lse[2], delta[2], mu[2], eps[2], cterm[2];
      };
      int g = 0, kact = 0;
      bool ok = true;
      FItem it;
      for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
        if (it.n_sub == 0) continue;
        // The own tiles are single-buffered: every MMA that reads the previous item's must be complete.
        const int oset = kact % C::OWN_BUFS, ouse = kact / C::OWN_BUFS;  // set of own tiles and how often it was used
        if (ouse > 0 && !mbar_wait_backoff(own_free + oset, (ouse - 1) & 1, ab, kAbortBwdOwn)) break;
        if (lane == 0) {
          unsigned char* dst = sOwn + oset * C::OWN_SET_BYTES;
          uint64_t* full = own_full + oset;
          mbar_expect_tx(full, C::N_OWN * C::OWN_BYTES);
          tma_load_4d(dst + C::SLOT_K * C::OWN_BYTES, &maps.k, full, 0, it.own0, it.h, it.b);
          tma_load_4d(dst + C::SLOT_V * C::OWN_BYTES, &maps.v, full, 0, it.own0, it.h, it.b);
          if constexpr (HAS_GT) {
            tma_load_4d(dst + C::SLOT_TK * C::OWN_BYTES, &maps.tk, full, 0, it.own0, it.h, it.b);
            tma_load_4d(dst + C::SLOT_TV * C::OWN_BYTES, &maps.tv, full, 0, it.own0, it.h, it.b);
          }
        }
        const size_t stat_off = (size_t)it.bh * L;
        // lane l holds the statistics of queries 2l, 2l+1 of a sub-tile; fetched one sub-tile ahead of their use
        auto load_stats = [&](int s, Stat& r) {
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            r.lse[e] = INFINITY, r.delta[e] = r.mu[e] = r.eps[e] = r.cterm[e] = 0.f;
            const int i = it.loop_begin + s * BL + 2 * lane + e;
            if (s < it.n_sub && i < L) {
              r.lse[e] = a.lse[stat_off + i];
              r.delta[e] = a.delta[stat_off + i];
              if constexpr (HAS_GT) {
                r.mu[e] = a.mu[stat_off + i];
                r.eps[e] = a.eps[stat_off + i];
                r.cterm[e] = a.cterm[stat_off + i];
              }
            }
          }
        };
        // One sub-tile: its tiles, the loads of the next one's statistics, and its own, which arrived meanwhile.  (Two names that
        // take turns: a copy from one to the other would wait for the loads, and the next tiles with it.)
        auto sub_tile = [&](int s, const Stat& cur, Stat& nxt) -> bool {
          const int st = g % STAGES;
          if (!mbar_wait_backoff<32>(loop_empty + st, ((g / STAGES) & 1) ^ 1, ab, kAbortBwdLoopEmpty)) return false;
          const int l0 = it.loop_begin + s * BL;
          if (lane == 0) {
            unsigned char* base = sRing + st * C::STAGE_BYTES;
            mbar_expect_tx(loop_full + st, C::STAGE_BYTES);
            tma_load_4d(base + C::SLOT_Q * C::LOOP_BYTES, &maps.q, loop_full + st, 0, l0, it.h, it.b);
            if constexpr (HAS_GT) tma_load_4d(base + C::SLOT_TQ * C::LOOP_BYTES, &maps.tq, loop_full + st, 0, l0, it.h, it.b);
            if constexpr (!C::TWO_RINGS) {
              if constexpr (HAS_GO) tma_load_4d(base + C::SLOT_GO * C::LOOP_BYTES, &maps.go, loop_full + st, 0, l0, it.h, it.b);
              if constexpr (HAS_GT) tma_load_4d(base + C::SLOT_G * C::LOOP_BYTES, &maps.g, loop_full + st, 0, l0, it.h, it.b);
            }
          }
          const int gst = g % GSTAGES;
          if constexpr (C::TWO_RINGS) {
            if (!mbar_wait_backoff<32>(g_empty + gst, ((g / GSTAGES) & 1) ^ 1, ab, kAbortBwdLoopEmpty)) return false;
            if (lane == 0) {
              unsigned char* base = sG + gst * C::G_STAGE_BYTES;
              mbar_expect_tx(g_full + gst, C::G_STAGE_BYTES);
              tma_load_4d(base + C::SLOT_G * C::LOOP_BYTES, &maps.g, g_full + gst, 0, l0, it.h, it.b);
              tma_load_4d(base + C::SLOT_GO * C::LOOP_BYTES, &maps.go, g_full + gst, 0, l0, it.h, it.b);
            }
          }
          load_stats(s + 1, nxt);
          // negated and stored pairwise for the packed arithmetic:
          //   float4 A = (-lse0, -lse1, -mu0, -mu1), float4 B = (-eps0, -eps1, -sub0, -sub1)
          float4* dst = sStat + (gst * (BL / 2) + lane) * 2;
          dst[0] = make_float4(-cur.lse[0], -cur.lse[1], -cur.mu[0], -cur.mu[1]);
          dst[1] = make_float4(-cur.eps[0], -cur.eps[1], -(cur.delta[0] + cur.cterm[0] + cur.eps[0] * cur.mu[0]),
                               -(cur.delta[1] + cur.cterm[1] + cur.eps[1] * cur.mu[1]));
          __syncwarp();
          if (lane == 0) mbar_arrive(stat_full + gst);
          ++g;
          return true;
        };
        Stat s0, s1;
        load_stats(0, s0);
        for (int s = 0; ok && s < it.n_sub; s += 2) {
          ok = sub_tile(s, s0, s1);
          if (ok && s + 1 < it.n_sub) ok = sub_tile(s + 1, s1, s0);
        }
        ++kact;
      }
    } else {
      // The issuing warps stay converged and let one lane issue (mbar_wait_warp), at most eight instructions in a row: the operands
      // of sixteen are computed ahead, and those uniform registers spill.
      {
        constexpr uint32_t idesc_sc = make_idesc(Fmt<T>::kIdesc, OWN, BL, 0, 0);       // 128 x 64 scores
        constexpr uint32_t idesc_sc2 = make_idesc(Fmt<T>::kIdesc, OWN, 2 * BL, 0, 0);  // 128 x 128: [S | tS]
        constexpr uint32_t idesc_kv = make_idesc(Fmt<T>::kIdesc, OWN, D, 0, 1);        // dK, dV: 128 x 64, B MN-major
        constexpr uint32_t idesc_dq = make_idesc(Fmt<T>::kIdesc, BL, D, 1, 1);         // dQ: 64 x 64, A and B MN-major
        // MN-major operands made of one 64-element chunk: the leading offset is not used (any value), 8-row groups 1024 B
        constexpr uint32_t kLoMN = (uint32_t)(8192 >> 4) << 16;
        constexpr uint32_t OWN16 = C::OWN_BYTES >> 4, LOOP16 = C::LOOP_BYTES >> 4, OUT16 = C::OUT_BYTES >> 4,
                           STAGE16 = C::STAGE_BYTES >> 4;
        const uint32_t own_k0 = kDescLo | (smem_u32(sOwn) >> 4);    // own tiles (first set) as K-major A operands
        const uint32_t own_mn0 = kLoMN | (smem_u32(sOwn) >> 4);     // ... as MN-major B operands (dQ)
        constexpr uint32_t OWNSET16 = C::OWN_SET_BYTES >> 4;
        const uint32_t ring_k = kDescLo | (smem_u32(sRing) >> 4);  // streamed tiles as K-major B operands (scores)
        const uint32_t ring_mn = kLoMN | (smem_u32(sRing) >> 4);   // ... as MN-major B operands (dK, dV)
        constexpr uint32_t GSTAGE16 = C::G_STAGE_BYTES >> 4;       // G and gO: a ring of their own, or beside Q
        const uint32_t gring_k = kDescLo | (smem_u32(sG) >> 4), gring_mn = kLoMN | (smem_u32(sG) >> 4);
        const uint32_t out_k = kDescLo | (smem_u32(sOut) >> 4);    // elementwise results as K-major A operands (dK, dV)
        const uint32_t out_mn = kLoMN | (smem_u32(sOut) >> 4);     // ... as MN-major A operands (dQ)
        int g = 0, kact = 0;
        bool ok = true;
        FItem it;
        if (warp == 1) {
          // ---------------------------------------------------------------- scores
          uint32_t own_k = own_k0;  // this item's set
          auto score = [&](uint32_t col, uint32_t own_slot, uint32_t b_lo, uint32_t id, bool first) {
            const uint32_t a_lo = own_k + own_slot * OWN16;
            if (first)
              umma_ss_lo<false>(tmem + col, a_lo, b_lo, id);
            else
              umma_ss_lo<true>(tmem + col, a_lo, b_lo, id);
#pragma unroll
            for (int ks = 1; ks < HD / 16; ++ks) umma_ss_lo<true>(tmem + col, a_lo + ks * 2, b_lo + ks * 2, id);
          };
          for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
            if (it.n_sub == 0) continue;
            const int oset = kact % C::OWN_BUFS;
            if (!mbar_wait_warp(own_full + oset, (kact / C::OWN_BUFS) & 1, ab, kAbortBwdOwn)) break;
            own_k = own_k0 + oset * OWNSET16;
            for (int s = 0; s < it.n_sub; ++s, ++g) {
              const int st = g % STAGES;
              if (!mbar_wait_warp(loop_full + st, (g / STAGES) & 1, ab, kAbortBwdLoopFull) ||
                  (g > 0 && !mbar_wait_warp(s_free, (g - 1) & 1, ab, kAbortBwdSFull))) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint32_t lp = ring_k + st * STAGE16;
              const uint32_t lg = C::TWO_RINGS ? gring_k + (g % GSTAGES) * GSTAGE16 : lp;
              auto from_q = [&]() {
                if constexpr (HAS_GT) {
                  score(C::COL_S, C::SLOT_K, lp + C::SLOT_Q * LOOP16, idesc_sc2, true);    // [S | tS] = K [Q ; tQ]^T
                  score(C::COL_TS, C::SLOT_TK, lp + C::SLOT_Q * LOOP16, idesc_sc, false);  // tS += tK Q^T
                } else {
                  score(C::COL_S, C::SLOT_K, lp + C::SLOT_Q * LOOP16, idesc_sc, true);  // S = K Q^T
                }
              };
              auto from_g = [&]() {
                if constexpr (HAS_GT) {
                  score(C::COL_E, C::SLOT_V, lg + C::SLOT_G * LOOP16, HAS_GO ? idesc_sc2 : idesc_sc, true);  // E = V G^T; [E | FP] = V [G ; gO]^T
                  score(C::COL_FP, C::SLOT_TV, lg + C::SLOT_G * LOOP16, idesc_sc, !HAS_GO);                  // FP (+)= tV G^T
                } else {
                  score(C::COL_FP, C::SLOT_V, lg + C::SLOT_GO * LOOP16, idesc_sc, true);  // FP = V gO^T
                }
                tc_commit(s_full);
                tc_commit(C::TWO_RINGS ? g_empty + g % GSTAGES : loop_empty + st);
                if (s == it.n_sub - 1) tc_commit(own_free + oset);
              };
              if constexpr (C::TWO_RINGS) {
                if (elect_one()) {
                  from_q();
                  tc_commit(loop_empty + st);
                }
                if (!mbar_wait_warp(g_full + g % GSTAGES, (g / GSTAGES) & 1, ab, kAbortBwdLoopFull)) {
                  ok = false;
                  break;
                }
                tc_fence_after();
                if (elect_one()) from_g();
              } else {
                if (elect_one()) from_q();
                if (elect_one()) from_g();
              }
            }
            if (!ok) break;
            ++kact;
          }
        } else if (warp == 2) {
          // ---------------------------------------------------------------- dK, dV
          // out (+)= result tile (A, K-major: 128 keys x 64 queries) x streamed tile (B, MN-major: 64 queries x 64)
          uint32_t ob16 = 0;  // result buffer of the sub-tile, in 16-byte units
          auto outer = [&](uint32_t col, uint32_t out_slot, uint32_t b_lo, uint32_t accumulate) {
            const uint32_t a_lo = out_k + ob16 + out_slot * OUT16;
            mma_ss_dyn(tmem + col, a_lo, b_lo, idesc_kv, accumulate);
#pragma unroll
            for (int ks = 1; ks < BL / 16; ++ks) umma_ss_lo<true>(tmem + col, a_lo + ks * 2, b_lo + ks * 128, idesc_kv);
          };
          // out (+)= packed operand (A, TMEM: 8 columns per 16 queries) x streamed tile (B, MN-major)
          auto outer_t = [&](uint32_t col, uint32_t a_col, uint32_t b_lo, uint32_t accumulate) {
            umma_ts_lo_dyn(tmem + col, tmem + a_col, b_lo, idesc_kv, accumulate);
#pragma unroll
            for (int ks = 1; ks < BL / 16; ++ks) umma_ts_lo<true>(tmem + col, tmem + a_col + ks * 8, b_lo + ks * 128, idesc_kv);
          };
          for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
            if (it.n_sub == 0) continue;
            for (int s = 0; s < it.n_sub; ++s, ++g) {
              const int st = g % STAGES;
              if (!mbar_wait_warp(p_full + (g & 1), (g >> 1) & 1, ab, kAbortBwdPFull) ||
                  (s == 0 && kact > 0 && !mbar_wait_warp(acc_free, (kact - 1) & 1, ab, kAbortBwdDone))) {
                ok = false;
                break;
              }
              tc_fence_after();
              const int ob = g % C::N_OBUF;
              ob16 = ob * (C::OBUF_BYTES >> 4);
              const uint32_t lp = ring_mn + st * STAGE16;
              const uint32_t lg = C::TWO_RINGS ? gring_mn + (g % GSTAGES) * GSTAGE16 : lp;
              const uint32_t acc = s > 0;
              // dV first: the stage of G and gO (two stages where they have a ring of their own) and the packed A and P come free
              // earlier, which the next scores and the elementwise threads wait for
              if (elect_one()) {
                if constexpr (HAS_GT) {
                  outer_t(C::COL_DV, C::COL_AV, lg + C::SLOT_G * LOOP16, acc);  // dV += A^T G
                  if constexpr (HAS_GO) outer_t(C::COL_DV, C::COL_P, lg + C::SLOT_GO * LOOP16, 1);  // dV += P^T gO
                } else {
                  outer_t(C::COL_DV, C::COL_P, lg + C::SLOT_GO * LOOP16, acc);  // dV += P^T gO
                }
                if constexpr (C::TWO_RINGS) tc_commit(g_empty + g % GSTAGES);
                tc_commit(av_free);
              }
              if (elect_one()) {
                outer(C::COL_DK, C::OUT_GS, lp + C::SLOT_Q * LOOP16, acc);                        // dK += gS^T Q
                if constexpr (HAS_GT) outer(C::COL_DK, C::OUT_GT, lp + C::SLOT_TQ * LOOP16, 1);  // dK += gtS^T tQ
                tc_commit(loop_empty + st);
                tc_commit(out_free + ob);
                if (s == it.n_sub - 1) tc_commit(done);
              }
            }
            if (!ok) break;
            ++kact;
          }
        } else {
          // ---------------------------------------------------------------- dQ of the sub-tile
          // dQ (+)= result tile (A, MN-major: 64 queries x 128 keys) x own tile (B, MN-major: 128 keys x 64)
          uint32_t ob16 = 0;
          uint32_t own_mn = own_mn0;  // this item's set
          auto inner = [&](uint32_t col, uint32_t out_slot, uint32_t own_slot, bool first) {
            const uint32_t a_lo = out_mn + ob16 + out_slot * OUT16, b_lo = own_mn + own_slot * OWN16;
            if (first)
              umma_ss_lo<false>(tmem + col, a_lo, b_lo, idesc_dq);
            else
              umma_ss_lo<true>(tmem + col, a_lo, b_lo, idesc_dq);
#pragma unroll
            for (int ks = 1; ks < OWN / 16; ++ks) umma_ss_lo<true>(tmem + col, a_lo + ks * 128, b_lo + ks * 128, idesc_dq);
          };
          for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
            if (it.n_sub == 0) continue;
            own_mn = own_mn0 + (kact % C::OWN_BUFS) * OWNSET16;
            for (int s = 0; s < it.n_sub; ++s, ++g) {
              if (!mbar_wait_warp(p_full + (g & 1), (g >> 1) & 1, ab, kAbortBwdPFull) ||
                  (g >= 1 && !mbar_wait_warp(dq_free, (g - 1) & 1, ab, kAbortBwdDone))) {
                ok = false;
                break;
              }
              tc_fence_after();
              const int ob = g % C::N_OBUF;
              ob16 = ob * (C::OBUF_BYTES >> 4);
              const uint32_t col = C::COL_DQ;
              if (elect_one()) {
                inner(col, C::OUT_GS, C::SLOT_K, true);                       // dQ = gS K
              }
              if (elect_one()) {
                if constexpr (HAS_GT) inner(col, C::OUT_GT, C::SLOT_TK, false);  // dQ += gtS tK
                tc_commit(dq_full);
                tc_commit(out_free + ob);
                if (s == it.n_sub - 1) tc_commit(own_free + kact % C::OWN_BUFS);
              }
            }
            if (!ok) break;
            ++kact;
          }
        }
      }
    }
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    // ------------------------------------------------------------------ elementwise warpgroups
    const int wg = (warp - 4) >> 2;  // 0 / 1: query columns [32 wg, 32 wg + 32) of every sub-tile
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;  // key row of the own tile <-> TMEM lane
    const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + 32 * wg;
    const float2 c2 = make_float2(a.sm_scale * kLog2e, a.sm_scale * kLog2e);
    const float2 sc2 = make_float2(a.sm_scale, a.sm_scale);
    // this thread's row of the result tiles: 16-byte chunk c (8 queries) sits at position c ^ (row & 7)
    const uint32_t out_row = smem_u32(sOut) + row * 128;
    const uint32_t sw = (uint32_t)(row & 7);
    bool alive = true;
    int g = 0, kact = 0;
    FItem it;

    auto store_row = [&](void* gptr, int bh, int own_idx, const uint32_t (&r0)[32], const uint32_t (&r1)[32], float mul) {
      if (own_idx >= L) return;
      T* gp = reinterpret_cast<T*>(gptr) + ((size_t)bh * L + own_idx) * HD;
#pragma unroll
      for (int x = 0; x < 4; ++x)
        reinterpret_cast<uint4*>(gp)[x] = make_uint4(
            Elem<T>::pack(__uint_as_float(r0[8 * x]) * mul, __uint_as_float(r0[8 * x + 1]) * mul),
            Elem<T>::pack(__uint_as_float(r0[8 * x + 2]) * mul, __uint_as_float(r0[8 * x + 3]) * mul),
            Elem<T>::pack(__uint_as_float(r0[8 * x + 4]) * mul, __uint_as_float(r0[8 * x + 5]) * mul),
            Elem<T>::pack(__uint_as_float(r0[8 * x + 6]) * mul, __uint_as_float(r0[8 * x + 7]) * mul));
      if constexpr (HD == 32) return;
#pragma unroll
      for (int x = 0; x < 4; ++x)
        reinterpret_cast<uint4*>(gp)[4 + x] = make_uint4(
            Elem<T>::pack(__uint_as_float(r1[8 * x]) * mul, __uint_as_float(r1[8 * x + 1]) * mul),
            Elem<T>::pack(__uint_as_float(r1[8 * x + 2]) * mul, __uint_as_float(r1[8 * x + 3]) * mul),
            Elem<T>::pack(__uint_as_float(r1[8 * x + 4]) * mul, __uint_as_float(r1[8 * x + 5]) * mul),
            Elem<T>::pack(__uint_as_float(r1[8 * x + 6]) * mul, __uint_as_float(r1[8 * x + 7]) * mul));
    };

    auto store_zeros = [&](int bh, int own_idx) {  // nothing attends these keys (they are all padding): the gradients are zero
      uint32_t z[32];
#pragma unroll
      for (int x = 0; x < 32; ++x) z[x] = 0u;
      store_row(wg == 0 ? a.dk : a.dv, bh, own_idx, z, z, 0.f);
    };
    if (CUT && a.mask.kind == JVPFA_MASK_KVLEN) {  // (weightless on the line: dealt to all CTAs alike)
      for (int w = cta; w < n_items; w += G) {
        const int bh = w / n_own_tiles, own0 = (w - bh * n_own_tiles) * OWN;
        if (own0 >= valid_keys(bh / a.H)) store_zeros(bh, own0 + row);
      }
    }

    for (int walk = begin_items(); alive && get_item(walk, it); ++walk) {
      const int own_idx = it.own0 + row;
      if (it.n_sub == 0) {
        if (!CUT) store_zeros(it.bh, own_idx);
        continue;
      }
      const int n_valid = valid_keys(it.b);
      const uint32_t* bcol = nullptr;  // packed boolean mask: this key's bits over the queries
      if (MK == 1 && a.mask_bits_t != nullptr)
        bcol = mask_bit_col(a.mask_bits_t, a.mask, mask_head(a.mask, it.b, it.h, a.H), min(own_idx, L - 1), L);
      // What the mask holds for this key and the 32 queries from l0 on (MK = 1: a bit each, packed one word, else byte by byte;
      // MK = 2: the bias elements, 16 bit each, of the tensors' type; two neighbouring lanes take two keys' elements of 16 queries each and
      // change half of them when they are used: half the loads and half the registers of an element at a time (us on a B200 for
      // H37 L2048: through O 238 -> 200, through tO 304 -> 252, both 352 -> 282).  Requested a sub-tile ahead, when the scores of this one have
      // left their registers: behind that the scores of the next are long there, and the loads would be waited for.  Indices are
      // clamped into the tensor; what lies outside is switched off by col_hi and by lse = +inf of the padding queries.
      uint32_t next_live = 0xffffffffu, braw[MK == 2 ? 16 : 1];
      auto fetch_mask = [&](int l0) {
        if (MK == 1 && bcol != nullptr) {
          next_live = l0 < L ? ldg_nc_u32(bcol + (a.mask.stride[2] ? l0 >> 5 : 0)) : 0u;
        } else if constexpr (MK == 2) {
          const long long step = a.mask.stride[2] * 2;  // to the next query; the last one's elements stand for those beyond
          // (not ragged: L is a multiple of 16 and so is q0, and the 16 queries are all there or none is; else the last pair of an odd length ends in
          // its row's padding)
          const int q0 = l0 + 16 * (lane & 1);
          const unsigned char* el = reinterpret_cast<const unsigned char*>(a.mask.ptr) +
                                    ((long long)it.b * a.mask.stride[0] + (long long)it.h * a.mask.stride[1] +
                                     min(own_idx - (lane & 1), RAG ? (L - 1) & ~1 : L - 2)) * 2 +
                                    min(q0, RAG ? L - 1 : L - 16) * step;
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            braw[x] = ldg_nc_u32(el);
            if (!RAG || q0 + x + 1 < L) el += step;
          }
        } else if constexpr (MK == 1) {
          const long long step = a.mask.stride[2];
          const unsigned char* el = reinterpret_cast<const unsigned char*>(a.mask.ptr) + (long long)it.b * a.mask.stride[0] +
                                    (long long)it.h * a.mask.stride[1] + (long long)min(own_idx, L - 1) * a.mask.stride[3] + min(l0, L - 1) * step;
          const int left = L - 1 - l0;
          next_live = 0u;
#pragma unroll
          for (int col = 0; col < 32; ++col) {
            next_live |= (ldg_nc_u8(el) != 0u ? 1u : 0u) << col;
            if (col < left) el += step;
          }
        }
      };
      if constexpr (MK != 0) fetch_mask(it.loop_begin + 32 * wg);
      for (int s = 0; s < it.n_sub; ++s, ++g) {
        const int st = g % GSTAGES;  // of the statistics
        const int l0 = it.loop_begin + s * BL + 32 * wg;  // first query of this group's columns
        uint32_t live = next_live;  // MK = 1: bit col = the mask lets query l0 + col attend this key
        // A look at a barrier takes 100 to 170 cycles also when its phase is long complete, so the looks are taken together, or ahead
        // of their need and under other work: three of four in a row were 540 of a sub-tile's 2760 cycles (through tO).
        const int ob = g % C::N_OBUF, use = g / C::N_OBUF;
        const uint32_t stat_ok = mbar_test(stat_full + st, (g / GSTAGES) & 1), s_ok = mbar_test(s_full, g & 1);
        const uint32_t out_ok = use == 0 ? 1u : mbar_test(out_free + ob, (use - 1) & 1);
        if ((!stat_ok && !mbar_wait(stat_full + st, (g / GSTAGES) & 1, ab, kAbortBwdLoopFull)) ||
            (!s_ok && !mbar_wait(s_full, g & 1, ab, kAbortBwdSFull))) {
          alive = false;
          break;
        }
        tc_fence_after();
        uint32_t bias[MK == 2 ? 16 : 1];
        if constexpr (MK == 2) {  // this lane's key, queries 2 x and 2 x + 1 in bias[x]; lane pairs: even keys' elements are the low halves
          const bool odd = lane & 1;
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const uint32_t lo = __byte_perm(braw[2 * x], braw[2 * x + 1], 0x5410), hi = __byte_perm(braw[2 * x], braw[2 * x + 1], 0x7632);
            const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
            bias[x] = odd ? other : lo;
            bias[8 + x] = odd ? hi : other;
          }
        }
        uint32_t sv[32], fp[32], ts[HAS_GT ? 32 : 1], ev[HAS_GT ? 32 : 1];
        tmem_ld32(tbase + C::COL_S, sv);
        tmem_ld32(tbase + C::COL_FP, fp);
        if constexpr (HAS_GT) {
          tmem_ld32(tbase + C::COL_TS, ts);
          tmem_ld32(tbase + C::COL_E, ev);
        }
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(s_free);
        // The products of the sub-tile that used this result buffer last must have read it.
        if (!out_ok && !mbar_wait(out_free + ob, (use - 1) & 1, ab, kAbortBwdPFull)) {
          alive = false;
          break;
        }
        // (key j = own_idx, query i = l0 + col) is dead if j >= n_valid, or causal and j > i: columns in [col_lo, col_hi) live
        int col_lo = 0, col_hi = 32;
        if (own_idx >= n_valid) col_hi = 0;
        if (causal) col_lo = own_idx - l0;
        const float4* stat = sStat + (st * (BL / 2) + 16 * wg) * 2;
        uint32_t pk_gs[16], pk_gt[HAS_GT ? 16 : 1], pk_av[HAS_GT ? 16 : 1], pk_p[HAS_GO ? 16 : 1];
        // One column pair: p from the scores and the row statistics, then the 16-bit operands.  MASKED: columns
        // outside [col_lo, col_hi) get p = 0.  Most sub-tiles have no dead pair for any thread of the warp and take
        // the variant without the comparisons and selects.
        auto pair = [&](int x, auto masked_c) {
          constexpr bool MASKED = decltype(masked_c)::value != 0;
          const int col = 2 * x;
          const float4 sa = stat[2 * x], sb = stat[2 * x + 1];
          const float2 nl = make_float2(sa.x, sa.y), nmu = make_float2(sa.z, sa.w);
          const float2 neps = make_float2(sb.x, sb.y), nsub = make_float2(sb.z, sb.w);
          float2 xs = __ffma2_rn(ff(sv[2 * x], sv[2 * x + 1]), c2, nl);
          if constexpr (MK == 2)  // scores are in log2 units: + bias * log2(e)
            xs = __ffma2_rn(unpack2<T>(bias[x]), make_float2(kLog2e, kLog2e), xs);
          float2 p = make_float2(fast_exp2(xs.x), fast_exp2(xs.y));
          if constexpr (MASKED) {
            if constexpr (MK == 1) {
              if (!((live >> col) & 1u)) p.x = 0.f;
              if (!((live >> (col + 1)) & 1u)) p.y = 0.f;
            } else {
              if (!(col >= col_lo && col < col_hi)) p.x = 0.f;
              if (!(col + 1 >= col_lo && col + 1 < col_hi)) p.y = 0.f;
            }
          }
          const float2 u = __fadd2_rn(ff(fp[2 * x], fp[2 * x + 1]), nsub);
          if constexpr (HAS_GT) {
            const float2 tm = __ffma2_rn(ff(ts[2 * x], ts[2 * x + 1]), sc2, nmu);
            const float2 eb = __fadd2_rn(ff(ev[2 * x], ev[2 * x + 1]), neps);
            const float2 av = __fmul2_rn(p, tm);
            const float2 gt = __fmul2_rn(p, eb);
            const float2 gs = __fmul2_rn(p, __ffma2_rn(eb, tm, u));
            pk_gs[x] = Elem<T>::pack(gs.x, gs.y);
            pk_gt[x] = Elem<T>::pack(gt.x, gt.y);
            pk_av[x] = Elem<T>::pack(av.x, av.y);
          } else {
            const float2 gs = __fmul2_rn(p, u);
            pk_gs[x] = Elem<T>::pack(gs.x, gs.y);
          }
          if constexpr (HAS_GO) pk_p[x] = Elem<T>::pack(p.x, p.y);
        };
        // Queries 8 c .. 8 c + 7 of this group (chunk 4 wg + c of the row) are written as soon as they are there.
        uint32_t av_ok = 0u;
        auto chunk = [&](int c, auto masked_c) {
#pragma unroll
          for (int x = 4 * c; x < 4 * c + 4; ++x) pair(x, masked_c);
          const uint32_t off = out_row + ob * C::OBUF_BYTES + (((uint32_t)(4 * wg + c) ^ sw) << 4);
          sts_v4(off + C::OUT_GS * C::OUT_BYTES, pk_gs[4 * c], pk_gs[4 * c + 1], pk_gs[4 * c + 2], pk_gs[4 * c + 3]);
          if constexpr (HAS_GT) sts_v4(off + C::OUT_GT * C::OUT_BYTES, pk_gt[4 * c], pk_gt[4 * c + 1], pk_gt[4 * c + 2], pk_gt[4 * c + 3]);
          if (c == 2) av_ok = g == 0 ? 1u : mbar_test_quiet(av_free, (g - 1) & 1);
        };
        if constexpr (MK == 1) {  // the index range (key padding of the own tile) joins the mask bits
          const int lo = max(col_lo, 0), hi = min(col_hi, 32);
          live &= hi > lo ? ((hi - lo >= 32 ? 0xffffffffu : ((1u << (hi - lo)) - 1u)) << lo) : 0u;
        }
        if (__any_sync(0xffffffffu, MK == 1 ? live != 0xffffffffu : (col_lo > 0 || col_hi < 32))) {
#pragma unroll
          for (int c = 0; c < 4; ++c) chunk(c, IntC<1>{});
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) chunk(c, IntC<0>{});
        }
        if constexpr (MK != 0) fetch_mask(l0 + BL);  // (behind the last one too: else this one's would have to be kept)
        // A and P go to their TMEM columns (this group's 32 queries = 16 packed columns) once the previous
        // sub-tile's dV products have read them
        if (!av_ok && !mbar_wait(av_free, (g - 1) & 1, ab, kAbortBwdPFull)) {
          alive = false;
          break;
        }
        tc_fence_after();  // (behind the look or the wait: the stores follow what av_free says has been read)
        {
          const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + 16 * wg;
          if constexpr (HAS_GT) tmem_st16(trow + C::COL_AV, pk_av);
          if constexpr (HAS_GO) tmem_st16(trow + C::COL_P, pk_p);
          fence_async_smem();
          tmem_wait_st();
        }
        tc_fence_before();
        mbar_arrive(p_full + (g & 1));
      }
      if (!alive) break;
      // item epilogue: group 0 stores dK, group 1 dV
      if (!mbar_wait(done, kact & 1, ab, kAbortBwdDone)) break;
      tc_fence_after();
      {
        uint32_t r0[32], r1[32];
        const uint32_t src = tmem + ((uint32_t)(quarter * 32) << 16) + (wg == 0 ? C::COL_DK : C::COL_DV);
        tmem_ld32(src, r0);
        tmem_ld32(src + 32, r1);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(acc_free);
        if (float* const to = share(walk, wg)) {
          uint4* p = reinterpret_cast<uint4*>(to) + row;
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            p[x * OWN] = make_uint4(r0[4 * x], r0[4 * x + 1], r0[4 * x + 2], r0[4 * x + 3]);
            p[(8 + x) * OWN] = make_uint4(r1[4 * x], r1[4 * x + 1], r1[4 * x + 2], r1[4 * x + 3]);
          }
        } else {
          store_row(wg == 0 ? a.dk : a.dv, it.bh, own_idx, r0, r1, wg == 0 ? a.sm_scale : 1.f);
        }
      }
      ++kact;
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    // ------------------------------------------------------------------ dQ read-back
    const int quarter = warp & 3;
    const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + C::COL_DQ;
    const uint32_t dqs = smem_u32(smem + C::OFF_DQS);
    int g = 0;
    bool alive = true;
    FItem it;
    // The 128 threads meet at a hardware barrier.  That is safe although it has no time limit: every decision to leave
    // the loop is taken from rb_ok, which one thread writes before a meeting and all read after it, so nobody can be
    // missing at the next one; and nothing between two meetings waits on another role.
    auto rb_meet = [&]() { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    for (int walk = begin_items(); alive && get_item(walk, it); ++walk) {
      if (it.n_sub == 0) continue;
      for (int s = 0; s < it.n_sub; ++s, ++g) {
        // one thread polls for the warpgroup (every polling warp is traffic on the shared-memory port)
        if (tid == 384) *rb_ok = mbar_wait(dq_full, g & 1, ab, kAbortBwdDone) ? 1 : 0;
        rb_meet();
        if (*rb_ok == 0) {
          alive = false;
          break;
        }
        tc_fence_after();
        uint32_t r0[32], r1[32];
        tmem_ld32(tbase, r0);
        tmem_ld32(tbase + 32, r1);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(dq_free);
        // An M = 64 accumulator: row 16 * quarter + l of the sub-tile is in lane l < 16 of this quarter.  The tile goes
        // to a staging area in shared memory and from there to the accumulation buffer as two TMA reductions (one
        // instruction each, coalesced and asynchronous) instead of sixteen vector reductions per thread.
        if (g > 0) {  // the previous sub-tile's reductions must have read the staging area
          if (tid == 384) bulk_wait_read();
          rb_meet();
        }
        if (lane < 16) {
          const int r = 16 * quarter + lane;
          const uint32_t rowa = dqs + r * 128, sw = (uint32_t)(r & 7);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            sts_v4(rowa + (((uint32_t)c ^ sw) << 4), r0[4 * c], r0[4 * c + 1], r0[4 * c + 2], r0[4 * c + 3]);
            if (HD > 32) sts_v4(rowa + 8192 + (((uint32_t)c ^ sw) << 4), r1[4 * c], r1[4 * c + 1], r1[4 * c + 2], r1[4 * c + 3]);
          }
        }
        fence_async_smem();
        rb_meet();
        if (tid == 384) {
          const int i0 = it.loop_begin + s * BL;
          if constexpr (parts) {
            tma_store_part_4d(&maps.dq, dqs, 0, i0, it.bh, it.own0 / OWN);
            if (HD > 32) tma_store_part_4d(&maps.dq, dqs + 8192, 32, i0, it.bh, it.own0 / OWN);
          } else {
            tma_reduce_add_4d(&maps.dq, dqs, 0, i0, it.h, it.b);
            tma_reduce_add_4d(&maps.dq, dqs + 8192, 32, i0, it.h, it.b);
          }
          bulk_commit();
        }
      }
    }
    if (tid == 384) bulk_wait_all();  // the reductions must have landed (and read shared memory) before the CTA ends
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) poison();
  if (warp == 0) {
    if (*abort_flag != 0) {
      // Something gave up: give copies and MMAs that may still be in flight time to land before the TMEM
      // columns go back to the allocator.
      const long long t0 = clock64();
      while (clock64() - t0 < (1ll << 22)) {
      }
    }
    tc_fence_after();
    tmem_dealloc(tmem, C::COLS_ALLOC);
  }
}

// dK and dV of the key tiles that were cut: the sum of their shares, in the order of the line.  Block x of 8 * (ctas - 1) looks at
// where CTA x / 8 + 1 begins: if that is the first cut of a key tile, the tile is this block's, an eighth of it (256 threads of 8
// columns; blocks 0-3 of the eight dK, the others dV).
template <typename T>
__device__ __forceinline__ void sum_shares(const jvpfa_bwd_args& a, const float* shares, int ctas, int block) {
  const int which = (block >> 2) & 1, row = threadIdx.x & 127, piece = 4 * (block & 3) + 2 * (threadIdx.x >> 7);
  const float4* p = reinterpret_cast<const float4*>(shares + kShareHead / 4) + piece * 128 + row;
  float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
  int item;
  if (!cut_shares(reinterpret_cast<const int2*>(shares), ctas, block / 8 + 1, &item, [&](int place) {
        const float4* q = p + (size_t)(2 * place + which) * (kShareFloats / 4);
        const float4 l = q[0], h = q[128];
        lo.x += l.x, lo.y += l.y, lo.z += l.z, lo.w += l.w;
        hi.x += h.x, hi.y += h.y, hi.z += h.z, hi.w += h.w;
      }))
    return;
  const int per_head = (a.L + 127) / 128, bh = item / per_head, key = (item - bh * per_head) * 128 + row;
  if (key >= a.L) return;
  if (4 * piece >= a.D) return;
  const float mul = which ? 1.f : a.sm_scale;
  T* out = reinterpret_cast<T*>(which ? a.dv : a.dk) + ((size_t)bh * a.L + key) * a.D + piece * 4;
  *reinterpret_cast<uint4*>(out) = make_uint4(Elem<T>::pack(lo.x * mul, lo.y * mul), Elem<T>::pack(lo.z * mul, lo.w * mul),
                                              Elem<T>::pack(hi.x * mul, hi.y * mul), Elem<T>::pack(hi.z * mul, hi.w * mul));
}

// What follows the single pass: dK and dV of cut key tiles (the first `cut` blocks), and dQ:
//   n_parts = 0: dq = T(scale * the accumulation buffer), 8 elements per thread
//   n_parts > 0: dq = T(scale * sum of the n_parts key tiles' shares of dQ, in their order), 4 elements per thread.  Bound by reading
//                them (B2 H12 L1024: 50 MB, most of it still in L2).
// CAUSAL: a query has a share of the key tiles up to its own.
template <typename T, bool CAUSAL>
__global__ void __launch_bounds__(256)
fused64_finish_kernel(const jvpfa_bwd_args a, const float* acc, long long n, int n_parts, const float* shares, int ctas, int cut) {
  behind_previous();
  if ((int)blockIdx.x < cut) return sum_shares<T>(a, shares, ctas, blockIdx.x);
  const long long i = (long long)((int)blockIdx.x - cut) * 256 + threadIdx.x;
  const float scale = a.sm_scale;
  if (n_parts == 0) {
    if (i >= n / 8) return;
    const float4 lo = reinterpret_cast<const float4*>(acc)[2 * i], hi = reinterpret_cast<const float4*>(acc)[2 * i + 1];
    reinterpret_cast<uint4*>(a.dq)[i] = make_uint4(Elem<T>::pack(lo.x * scale, lo.y * scale), Elem<T>::pack(lo.z * scale, lo.w * scale),
                                                   Elem<T>::pack(hi.x * scale, hi.y * scale), Elem<T>::pack(hi.z * scale, hi.w * scale));
    return;
  }
  const long long n4 = n / 4;
  if (i >= n4) return;
  const float4* p = reinterpret_cast<const float4*>(acc) + i;
  if constexpr (CAUSAL) n_parts = min(n_parts, (int)(4 * i / a.D % a.L) / 128 + 1);
  float4 s = __ldcs(p);
#pragma unroll 8
  for (int k = 1; k < n_parts; ++k) {
    const float4 x = __ldcs(p + k * n4);
    s.x += x.x, s.y += x.y, s.z += x.z, s.w += x.w;
  }
  reinterpret_cast<uint2*>(a.dq)[i] = make_uint2(Elem<T>::pack(s.x * scale, s.y * scale), Elem<T>::pack(s.z * scale, s.w * scale));
}

static int fused_sm_count() {
  static int cache[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!cache[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cache[dev] = n;
  }
  return cache[dev];
}

// Floats for a key tile's share of dQ, of every key tile: as many bytes as the (B, H, L, L) bias itself has, up to half a GiB; at
// head dimension 32 half as many, up to a quarter.  From 96 key tiles on: with fewer the two launches, of as many CTAs each, fill more of the 148 SMs.
// At head dimension 32, where key tiles are shared out, that only holds for short ones: both launches fit the SMs at once up to 74 tiles (through both,
// B2 H8 L512, 64 tiles: 18.8 / 21.2 us; B2 H10 L512, 80 tiles: 27.4 / 21.9; from L1024 on B1 H8 28 / 26 and fewer heads more), causal ones, of half the
// work, up to twice as many (B2 H12 L512 19.1 / 22.4, B1 H14 L778 23.9 / 24.9; B2 H17 L512, 136 tiles, 23.5 / 23.1; B2 H20 L512 26.2 / 23.7).
static long long bwd_parts_workspace(const jvpfa_bwd_args& a) {
  if ((a.dtype != JVPFA_BF16 && a.dtype != JVPFA_FP16) || a.impl == JVPFA_IMPL_GENERIC || (a.flags & JVPFA_SKIP_DKDV)) return 0;
  if (a.D > 64 || !tc5_head_dim(a.D, a.L) || !dq_parts(a)) return 0;
  if (a.mask.kind == JVPFA_MASK_BIAS) {
    // rows of whole 32-byte pieces, padded to them where the length does not fill them
    if (((a.L & 15) != 0 && a.mask.stride[2] < ((a.L + 15) & ~15)) || !tc5_mask_layout(a.mask, a.dtype, a.L)) return 0;
  } else if (a.mask.kind == JVPFA_MASK_BOOL) {
    if (a.mask_tile_live != nullptr || a.mask_tile_live_t != nullptr || a.mask_bits_t == nullptr) return 0;
  } else if (a.mask.kind == JVPFA_MASK_KVLEN) {
    return 0;  // (the sum would have to know which key tiles are all padding)
  }
  const long long key_tiles = (long long)((a.L + 127) / 128) * a.B * a.H;
  if (a.D == 32 ? a.L < 1024 && key_tiles < (a.mask.kind == JVPFA_MASK_CAUSAL ? 144 : 75) : key_tiles < 96) return 0;
  const long long bytes = key_tiles * a.L * a.D * 4;
  return bytes <= (a.D == 32 ? 1ll << 28 : 1ll << 29) ? bytes : 0;
}

// CTAs among which the key tiles' sub-tiles are shared out; 0: the key tiles are dealt whole.  Both in sub-tiles of the CTA that has
// the most: dealt whole, in rounds; shared out, an equal part, one more beginning of a key tile, and the time of the shares' way through
// the workspace: 2 sub-tiles (3 through O) and 2 (1) more where each CTA has two shares.  A twenty-fifth less is asked for: the last round
// of key tiles dealt whole has the memory to itself.  800 draws of B to 32, H to 40, L 256 to 4096 and every mask, where the shares' way at
// 2 (3) had these cut: 6 / 17 / 12 % of them were more than 2 % slower than whole tiles through O / tO / both (B3 H6 L640 through tO 27.3 whole, 32.6
// shared out), with this price 4 / 5 / 3 %, 12 % at most.  fp16 B3 H12 L1330 causal through O, left whole: 46 us, 51 shared out.
// Key padding: whole where the lengths are not known here.  With them 4 sub-tiles (5) and 3 more, and a twentieth less is asked for (pieces end
// anywhere in ragged entries, so more tiles are cut).  340 draws of B to 70, H to 16, L 256 to 4096 and lengths of L / 20 to L, through O /
// tO / both: 2 / 4 / 5 are more than 2 % slower than whole tiles, 7 % at most; by L alone, and with 2 (3) sub-tiles, every sixth was, 26 % at
// most (B2 H20 L1000, lengths 280 and 400, forward and backward 66 us whole, 74 shared out).
static int split_ctas(const jvpfa_bwd_args& a, int sms) {
  const int open = kOpen;
  const long long T = (a.L + 127) / 128, S = (a.L + 63) / 64, BH = (long long)a.B * a.H, items = T * BH;
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL, keys = a.mask.kind == JVPFA_MASK_KVLEN;
  if (keys && a.kv_len_host == nullptr) return 0;
  const long long G = items < sms ? items : sms;
  const HostLengths lengths(a.kv_len_host, a.B, a.L, keys && a.B <= kMaxSortedBatch && items > G);
  long long live = items;  // key tiles that are not all padding
  if (keys) {
    live = 0;
    for (int b = 0; b < a.B; ++b) live += lengths.tiles(b, 128) * a.H;
  }
  const long long subs = causal ? BH * (T * S - T * (T - 1)) : live * S, cost = subs + live * open;
  const long long ctas = subs / 4 < sms ? subs / 4 : sms;
  if (ctas < 2 || !cut_fits(items * (S + open), ctas)) return 0;  // (that many rounds need no cuts)
  const long long rounds = (items + G - 1) / G;
  if (rounds > (causal ? 8 : keys ? 16 : rounds)) return 0;  // (the lightest are dealt last and even out)
  const long long whole = causal ? most_loaded(items, G, 8, [&](long long w) { return S - 2 * (w / BH) + open; })
                          : keys ? most_loaded(items, G, 16, [&](long long w) { return lengths.tiles(w % BH / a.H, 128) > w / BH ? S + open : 0; })
                                 : rounds * (S + open);
  const int way = (a.gto ? 2 : 3) + (keys ? 2 : 0), more = keys ? 3 : a.gto ? 2 : 1, of = keys ? 20 : 25;
  const long long two = live < ctas ? live : ctas;  // CTAs that have two shares
  return (cost + (open + way) * ctas + more * two) * of < whole * ctas * (of - 1) ? (int)ctas : 0;
}

template <typename T, bool HAS_GO, bool HAS_GT, int MK, bool CUT, int HD, bool RAG>
static cudaError_t run_fused64_d(const jvpfa_bwd_args& a, const BwdFMaps& m, float* dq_acc, float* shares, int* status, int grid, cudaStream_t stream) {
  using C = BwdFCfg<HAS_GO, HAS_GT>;
  auto kern = bwd_tc5_fused64_kernel<T, HAS_GO, HAS_GT, MK, CUT, HD, RAG>;
  static SmemOptIn opt_in;
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return cudaErrorInvalidValue;
  return launch_behind(kern, grid, C::NTHREADS, C::SMEM_BYTES, stream, a, m, dq_acc, shares, status);
}

template <typename T, bool HAS_GO, bool HAS_GT, int MK, bool CUT>
static cudaError_t run_fused64(const jvpfa_bwd_args& a, const BwdFMaps& m, float* dq_acc, float* shares, int* status, int grid, cudaStream_t stream) {
  if constexpr (MK == 2) {
    if ((a.L & 15) != 0) {
      // (D = 64 through O alone: bwd_tc5_fused64_eligible takes no ragged bias)
      if (!HAS_GT || a.D == 32) return run_fused64_d<T, HAS_GO, HAS_GT, MK, CUT, 32, true>(a, m, dq_acc, shares, status, grid, stream);
      if constexpr (HAS_GT) return run_fused64_d<T, HAS_GO, HAS_GT, MK, CUT, 64, true>(a, m, dq_acc, shares, status, grid, stream);
    }
  }
  return a.D == 32 ? run_fused64_d<T, HAS_GO, HAS_GT, MK, CUT, 32, false>(a, m, dq_acc, shares, status, grid, stream)
                   : run_fused64_d<T, HAS_GO, HAS_GT, MK, CUT, 64, false>(a, m, dq_acc, shares, status, grid, stream);
}

template <typename T, bool HAS_GO, bool HAS_GT, int MK>
static int launch_fused64(const jvpfa_bwd_args& a, cudaStream_t stream) {
  using C = BwdFCfg<HAS_GO, HAS_GT>;
  int* status = tc5_status_device_ptr();
  if (!status) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  BwdFMaps m;
  const CUtensorMapDataType dt = Fmt<T>::kTma;
  const int64_t* st = a.in_stride;
  bool ok = encode_map4d(&m.k, dt, a.k, a.D, a.L, a.H, a.B, st, C::OWN) && encode_map4d(&m.v, dt, a.v, a.D, a.L, a.H, a.B, st, C::OWN) &&
            encode_map4d(&m.q, dt, a.q, a.D, a.L, a.H, a.B, st, C::BL);
  m.tk = m.tv = m.k;
  m.go = m.tq = m.g = m.q;
  if (HAS_GO) ok = ok && encode_map4d(&m.go, dt, a.go, a.D, a.L, a.H, a.B, nullptr, C::BL);
  if (HAS_GT)
    ok = ok && encode_map4d(&m.tk, dt, a.tk, a.D, a.L, a.H, a.B, st, C::OWN) && encode_map4d(&m.tv, dt, a.tv, a.D, a.L, a.H, a.B, st, C::OWN) &&
         encode_map4d(&m.tq, dt, a.tq, a.D, a.L, a.H, a.B, st, C::BL) && encode_map4d(&m.g, dt, a.gto, a.D, a.L, a.H, a.B, nullptr, C::BL);
  const bool parts = dq_parts(a);
  float* dq_acc = parts ? static_cast<float*>(a.workspace) : a.dq_accum;
  const int n_key_tiles = (a.L + C::OWN - 1) / C::OWN;
  ok = ok && (parts ? encode_map4d_f32(&m.dq, dq_acc, a.D, a.L, a.B * a.H, n_key_tiles, C::BL)
                    : encode_map4d_f32(&m.dq, dq_acc, a.D, a.L, a.H, a.B, C::BL));
  if (!ok) {
    set_last_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled(bwd fused64)");
    return JVPFA_ERR_CUDA;
  }
  const int sms = fused_sm_count();
  if (sms <= 0) {
    set_last_cuda_error(cudaErrorUnknown, "multiprocessor count");
    return JVPFA_ERR_CUDA;
  }
  const size_t n = (size_t)a.B * a.H * a.L * a.D;
  cudaError_t e = cudaSuccess;
  if (!parts && !(a.flags & JVPFA_DQ_ACCUM_IS_ZERO)) e = cudaMemsetAsync(a.dq_accum, 0, n * sizeof(float), stream);
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "cudaMemsetAsync(dq_accum)");
    return JVPFA_ERR_CUDA;
  }
  const long long n_items = (long long)n_key_tiles * a.B * a.H;
  int grid = (int)(n_items < sms ? n_items : sms);
  const long long used = parts ? bwd_parts_workspace(a) : 0;  // the split's workspace lies behind dQ's shares
  const int ctas = split_ctas(a, sms);
  float* shares = nullptr;
  if (ctas > 0 && a.workspace != nullptr && (reinterpret_cast<uintptr_t>(a.workspace) & 15u) == 0 &&
      a.workspace_bytes >= used + split_bytes(ctas)) {
    shares = reinterpret_cast<float*>(static_cast<char*>(a.workspace) + used);
    grid = ctas;
  }
  e = shares ? run_fused64<T, HAS_GO, HAS_GT, MK, true>(a, m, dq_acc, shares, status, grid, stream)
             : run_fused64<T, HAS_GO, HAS_GT, MK, false>(a, m, dq_acc, nullptr, status, grid, stream);
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch bwd_tc5_fused64");
    return JVPFA_ERR_CUDA;
  }
  const int cut = shares ? 8 * (ctas - 1) : 0;
  const long long per_block = parts ? 256 * 4 : 256 * 8;
  const long long blocks = cut + (a.flags & JVPFA_SKIP_DQ ? 0 : ((long long)n + per_block - 1) / per_block);
  if (blocks == 0) return JVPFA_OK;
  auto finish = parts && a.mask.kind == JVPFA_MASK_CAUSAL ? fused64_finish_kernel<T, true> : fused64_finish_kernel<T, false>;
  e = launch_behind(finish, (unsigned)blocks, 256, 0, stream, a, static_cast<const float*>(dq_acc), (long long)n,
                    parts ? n_key_tiles : 0, static_cast<const float*>(shares), ctas, cut);
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch fused64_finish");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <typename T>
static int launch_fused64_t(const jvpfa_bwd_args& a, cudaStream_t s) {
  const bool go = a.go != nullptr, gt = a.gto != nullptr;
  if (a.mask.kind == JVPFA_MASK_BIAS) {
    if (go && gt) return launch_fused64<T, true, true, 2>(a, s);
    if (gt) return launch_fused64<T, false, true, 2>(a, s);
    return launch_fused64<T, true, false, 2>(a, s);
  }
  if (a.mask.kind == JVPFA_MASK_BOOL) {
    if (go && gt) return launch_fused64<T, true, true, 1>(a, s);
    if (gt) return launch_fused64<T, false, true, 1>(a, s);
    return launch_fused64<T, true, false, 1>(a, s);
  }
  if (go && gt) return launch_fused64<T, true, true, 0>(a, s);
  if (gt) return launch_fused64<T, false, true, 0>(a, s);
  return launch_fused64<T, true, false, 0>(a, s);
}

}  // namespace tc5

// The single-pass kernel serves, where the caller provides a place for dQ:
//   D = 64, in dq_accum: index masks (none, causal, key padding), boolean masks that come without tile bitmaps, and through O alone a
//           bias of the tensors' type.  What goes there is summed in no fixed order, so masks and bias whose rows are not whole 16-byte
//           pieces, which kernels of a fixed order have always served, stay with those
//   D = 64 with a bias through tO, and D = 32, in the workspace, where dQ is summed in a fixed order: bwd_parts_workspace
bool bwd_tc5_fused64_eligible(const jvpfa_bwd_args& a) {
  const int k = a.mask.kind;
  if (tc5::dq_parts(a)) {
    const long long need = tc5::bwd_parts_workspace(a);
    return need > 0 && a.workspace != nullptr && a.workspace_bytes >= need && (reinterpret_cast<uintptr_t>(a.workspace) & 15u) == 0;
  }
  if (a.D != 64) return false;
  if (a.dq_accum == nullptr || (reinterpret_cast<uintptr_t>(a.dq_accum) & 15u) != 0) return false;
  if (k == JVPFA_MASK_NONE || k == JVPFA_MASK_CAUSAL || k == JVPFA_MASK_KVLEN) return true;
  if ((a.L & 15) != 0 || !tc5_mask_layout(a.mask, a.dtype, a.L)) return false;
  // A boolean mask without tile bitmaps (dense, or not looked at beforehand): with them the two-launch kernels, which
  // step over dead tiles, are the better choice.
  return k != JVPFA_MASK_BOOL || (a.mask_tile_live == nullptr && a.mask_tile_live_t == nullptr);
}

// What the launch can use: shares of dQ (needed for a bias through tO), and of dK and dV where key tiles are cut.
long long bwd_fused64_workspace(const jvpfa_bwd_args& a) {
  if ((a.dtype != JVPFA_BF16 && a.dtype != JVPFA_FP16) || a.impl == JVPFA_IMPL_GENERIC || a.D > 64 || (a.flags & JVPFA_SKIP_DKDV)) return 0;
  long long parts = 0;
  if (tc5::dq_parts(a)) {
    parts = tc5::bwd_parts_workspace(a);
    if (parts == 0) return 0;
  } else if (!bwd_tc5_fused64_eligible(a)) {
    return 0;
  }
  const int ctas = tc5::split_ctas(a, tc5::fused_sm_count());
  return parts + (ctas ? tc5::split_bytes(ctas) : 0);
}

int launch_bwd_tc5_fused64(const jvpfa_bwd_args& a, cudaStream_t s) {
  return a.dtype == JVPFA_BF16 ? tc5::launch_fused64_t<__nv_bfloat16>(a, s) : tc5::launch_fused64_t<__half>(a, s);
}

}  // namespace jvpfa
