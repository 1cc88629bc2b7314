// Fused primal (+ tangent) attention forward for head dimension 64 (bf16 / fp16) on tcgen05 / TMA /
// TMEM, organised so that the softmax never sits between two dependent MMAs of the same tile.
//
// One CTA per SM owns a PAIR of 128-row query tiles (256 query rows of one (batch, head)) and walks a
// static list of such pairs.  The two query tiles are two independent pipelines that share every
// K / tK / V / tV stage brought in by TMA (so each key tile is fetched once per 256 query rows):
//
//   issuer X (one thread per query tile):   [S | tS] = Q [K ; tK]^T (N=128) ; tS += tQ K^T (N=64)   -> s_full[X]
//                                           [O | tO'] += P [V | tV] (N=128) ; tO' += W V   (N=64)   -> pv_done[X], kv_empty
//   softmax X (one warpgroup per query tile, thread <-> query row <-> TMEM lane)
//
// P and W = P * tS * scale leave the softmax threads through SHARED memory (128-byte-swizzled K-major
// tiles, the layout TMA gives Q), not through TMEM.  The score accumulators are therefore free as soon
// as the softmax threads have copied them to registers (s_free[X]), and the issuer forms the scores of
// key tile j+1 while the softmax of tile j is still computing:
//
//   issue order per query tile:   S(0) ; S(1) PV(0) ; S(2) PV(1) ; ... ; PV(last)
//
// TMEM columns per query tile: S [64] | tS [64] | O [64] | tO' [64]; two query tiles = 512 columns.
// Online softmax with lazy rescaling: the running reference maximum is raised only when the tile maximum
// exceeds it by more than 2^8, and only then are O / tO' rescaled in TMEM (after PV of the previous tile
// has completed).  Row arithmetic uses packed fp32x2 instructions.
//
// Masks (template parameter MK): 0 = none / causal / key padding by index comparison; 1 = uint8 mask;
// 2 = additive bias of the element type; 3 = uint8 mask with the tile bitmap written by jvpfa_mask_tiles
// (one bit per 128-query x 64-key tile).  A softmax thread owns one query row, so its share of a boolean mask's tile is two words of
// packed bits or 64 bytes, which it fetches itself.  A bias comes by TMA, a 128 x 64 tile for each query tile; its 32 KiB of
// shared memory are what K and V with rings of their own save: K's stages are free when the scores exist, so two of each serve as
// three of both.  (Fetched by the threads, 32 rows of a warp at a time, the bias took the L1 longer than the tile's arithmetic: a key
// tile of a pair 3.05 us with tangents on a B200 where 1.5 without a mask; now 1.95.  B2 H12 L1024: with tangents 50 -> 36 us, without 33 -> 28.)
// With a bitmap the two query tiles may need different key tiles: the producer loads the union, and an
// issuer that does not use a loaded tile only releases it.
#include "tc5_common.cuh"

namespace jvpfa {
namespace tc5 {

template <bool DUAL, bool BIAS>
struct FwdPairCfg {
  static constexpr int D = 64;
  static constexpr int BM = 128;  // rows of one query tile
  static constexpr int NQ = 2;    // query tiles per CTA
  static constexpr int BN = 64;
  static constexpr int STAGES = BIAS ? 2 : 3;  // of K, V together, or with a bias of either
  static constexpr int NTHREADS = 384;  // warpgroup 0: TMA producer, two issuers, one idle warp; warpgroups 1, 2: softmax
  static constexpr int Q_BYTES = BM * D * 2;   // 16 KiB
  static constexpr int KV_BYTES = BN * D * 2;  // 8 KiB
  static constexpr int P_BYTES = BM * BN * 2;  // 16 KiB
  static constexpr int N_QT = DUAL ? 2 : 1;    // Q, tQ
  static constexpr int N_KV = DUAL ? 4 : 2;    // K, tK, V, tV
  static constexpr int N_P = DUAL ? 2 : 1;     // P, W
  static constexpr int HALF_BYTES = N_KV / 2 * KV_BYTES;               // K (, tK) or V (, tV) of a key tile
  static constexpr int STAGE_BYTES = BIAS ? HALF_BYTES : 2 * HALF_BYTES;  // from one stage to the next
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = NQ * N_QT * Q_BYTES;
  static constexpr int OFF_V = OFF_K + (BIAS ? STAGES : 1) * HALF_BYTES;
  static constexpr int OFF_P = OFF_K + STAGES * 2 * HALF_BYTES;
  static constexpr int B_BYTES = BM * BN * 2;  // a bias tile
  static constexpr int OFF_B = OFF_P + NQ * N_P * P_BYTES;
  static constexpr int TILE_BYTES = OFF_B + (BIAS ? NQ * B_BYTES : 0);
  static constexpr int OFF_ORDER = TILE_BYTES + 256;  // behind the barriers
  static constexpr int SMEM_BYTES = OFF_ORDER + kMaxSortedBatch + 1024;
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory budget");
  static constexpr int COL_S = 0;
  static constexpr int COL_TS = 64;
  static constexpr int COL_O = DUAL ? 128 : 64;
  static constexpr int COL_TO = 192;
  // Primal only: half of the columns are free, so P (packed 16-bit, 32 columns) stays in TMEM in a place of its
  // own and feeds the output MMAs as their A operand; nothing of P touches shared memory.
  static constexpr int COL_P = 128;
  static constexpr int COLS_PER_Q = 256;
  static constexpr int COLS_ALLOC = NQ * COLS_PER_Q;
};

struct FwdPairMaps {
  CUtensorMap q, tq, k, tk, v, tv;
  CUtensorMap bias;   // MK = 2; its own extents: a dimension that broadcasts has one entry
  CUtensorMap o, to;  // outputs, stored tile-wise from shared memory
};

// TMA store of one (64 x rows) tile from shared memory; rows past the tensor's extent are not written.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* smem_src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }



__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Makes this thread's shared-memory writes visible to the async proxy (the tensor core reads operands through it).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// One work item: two neighbouring 128-row query tiles of one (batch, head).  Per-query-tile fields are plain
// scalars picked with a select (arrays indexed by the query tile would live in local memory).
struct PairItem {
  int bh, b, h, m0, n_valid;
  int nt0, nt1;      // key tiles in range of each query tile (0: the tile has no row or no key)
  int last0, last1;  // index of the last key tile each query tile uses, -1 when it uses none
  int j0, n_load;    // key tiles to walk: [j0, n_load), up to max(nt0, nt1) where the item is not cut
  const unsigned long long *live0, *live1;  // MK == 3: the query tiles' words of the tile bitmap
  __device__ __forceinline__ int nt(int x) const { return x ? nt1 : nt0; }
  __device__ __forceinline__ int last(int x) const { return x ? last1 : last0; }
};

// Walks an item's key tiles in order: bit X of the result says that query tile X uses tile j.
template <int MK>
struct TileUse {
  const int nt0, nt1;
  const unsigned long long *l0, *l1;
  unsigned long long w0, w1;
  __device__ __forceinline__ explicit TileUse(const PairItem& i)
      : nt0(i.nt0), nt1(i.nt1), l0(i.live0), l1(i.live1), w0(0ull), w1(0ull) {}
  __device__ __forceinline__ int operator()(int j) {
    int m = (j < nt0 ? 1 : 0) | (j < nt1 ? 2 : 0);
    if constexpr (MK == 3) {
      if ((j & 63) == 0) {
        w0 = __ldg(l0 + (j >> 6));
        w1 = __ldg(l1 + (j >> 6));
      }
      m &= (int)((w0 >> (j & 63)) & 1ull) | ((int)((w1 >> (j & 63)) & 1ull) << 1);
    }
    return m;
  }
};

// ---- Pairs shared out among CTAs ----------------------------------------------------------------
// Dealt whole, 192 pairs (B2 H12 L2048) take two rounds of 148 CTAs where 1.3 rounds' worth of work is there, and 16 leave 132 SMs idle.
// With a workspace whole rounds of pairs are dealt whole (where all pairs are alike; else none), and the key tiles of the rest are one line
// that is cut into equal pieces (cut_begin); a pair that is cut leaves what each CTA has of it, O and tO' before the division and the
// rows' statistics, all fp32, in the workspace, and pair64_finish_kernel merges them in their order.  A pair's beginning counts as kPairOpen key tiles.
constexpr int kPairOpen = 2;
template <bool DUAL>
struct PairShare {  // floats: [query tile][16-byte piece of O, then of tO'][128 rows], then [128 rows]{maximum, sum, sum of W, 1: no key, no accumulators}
  static constexpr int PIECES = DUAL ? 32 : 16;
  static constexpr int TILE = (PIECES + 1) * 128 * 4;
  static constexpr int SIZE = 2 * TILE;
  static constexpr long long HEAD = 16 * 1024;  // bytes: where each CTA begins, {pair, key tile}
  static constexpr long long bytes(int ctas) { return HEAD + (long long)ctas * 2 * SIZE * 4; }
};
__device__ __forceinline__ int2 pair_begin(const jvpfa_fwd_args& a, int whole, int c, int G) {
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL;
  const int n_pairs = (a.L + 255) / 256, n_keys = (a.L + 63) / 64;
  auto first = [&](int b) {
    if (causal) return 4;
    return a.mask.kind == JVPFA_MASK_KVLEN ? (max(0, min(a.mask.kv_len[b], a.L)) + 63) / 64 : n_keys;
  };
  return cut_begin(
      a.mask.kind == JVPFA_MASK_KVLEN, a.B, a.H, n_pairs, causal ? 4 : 0, kPairOpen, whole, c, G, [&](int) { return n_pairs; }, first,
      [&](int b, int r) { return causal ? min(n_keys, 4 * r + 4) : first(b); });
}

template <typename T, bool DUAL, int MK, bool CUT>
__global__ void __launch_bounds__(384, 1)
fwd_tc5_pair64_kernel(const jvpfa_fwd_args a, const __grid_constant__ FwdPairMaps maps, float* shares, int whole, int* status) {
  using C = FwdPairCfg<DUAL, MK == 2>;
  constexpr int D = 64, BM = C::BM, BN = C::BN, STAGES = C::STAGES;
  constexpr bool BIAS = MK == 2;

  behind_previous();
  const bool dead_on_entry = *(volatile int*)status != 0;  // an earlier bounded wait gave up

  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  unsigned char* sQ = smem + C::OFF_Q;    // [query tile][Q, tQ]
  unsigned char* sK = smem + C::OFF_K;    // [stage][K, tK]; V, tV behind each stage's, or with a bias behind them all
  unsigned char* sV = smem + C::OFF_V;
  unsigned char* sB = smem + C::OFF_B;    // [query tile] bias
  unsigned char* sP = smem + C::OFF_P;    // [query tile][P, W]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::TILE_BYTES);
  uint64_t* q_full = bars + 0;
  uint64_t* q_empty = bars + 1;   // both issuers are through with the item's Q tiles
  uint64_t* kv_full = bars + 2;   // [STAGES]
  uint64_t* kv_empty = kv_full + STAGES;  // [STAGES], one arrival per issuer
  uint64_t* v_full = kv_empty + STAGES;   // BIAS: V's ring; kv_full and kv_empty are K's
  uint64_t* v_empty = v_full + (BIAS ? STAGES : 0);
  uint64_t* s_full = v_empty + (BIAS ? STAGES : 0);  // [2] per query tile from here on
  uint64_t* s_free = s_full + 2;          // the softmax threads hold the scores in registers
  uint64_t* p_full = s_free + 2;          // P / W are in shared memory
  uint64_t* pv_done = p_full + 2;         // the tile's output MMAs are complete
  uint64_t* o_free = pv_done + 2;         // the epilogue has read the item's accumulators
  uint64_t* wg_bar = o_free + 2;          // meeting point of a softmax warpgroup's 128 threads (bounded, unlike bar.sync)
  uint64_t* b_full = wg_bar + 2;          // BIAS: a tile of it is there
  uint64_t* b_empty = b_full + (BIAS ? 2 : 0);  // ... has been added
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(b_empty + (BIAS ? 2 : 0));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int L = a.L;
  const int BH = a.B * a.H;
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL;
  const int n_q_tiles = (L + BM - 1) / BM;
  const int n_pairs = (n_q_tiles + 1) / 2;
  const int n_items = n_pairs * BH;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  unsigned char* order = smem + C::OFF_ORDER;
  int* s_cut = reinterpret_cast<int*>(order);  // CUT: {pair, key tile} where this CTA and the next begin
  if constexpr (CUT) {
    if (warp < 2) {
      const int2 at = pair_begin(a, whole, cta + warp, G);
      if (lane == 0) {
        s_cut[2 * warp] = at.x, s_cut[2 * warp + 1] = at.y;
        if (warp == 0) reinterpret_cast<int2*>(shares)[cta] = at;
      }
    }
    __syncthreads();
  }
  const bool sorted = !CUT && a.mask.kind == JVPFA_MASK_KVLEN && a.B <= kMaxSortedBatch && n_items > G;
  if (sorted) {
    sort_batch(a.mask, a.B, order);
    __syncthreads();
  }

  // Item `walk` of this CTA.  Dealt whole, the round: items are ranked heaviest first (for causal masks the last pair is the longest) and
  // dealt in serpentine order.  Shared out: `whole` rounds, from -whole to -1, then the pairs from s_cut[0] on.
  auto begin_items = [&]() { return CUT ? -whole : 0; };
  auto get_item = [&](int walk, PairItem& it) -> bool {
    const int w = CUT ? (walk < 0 ? (walk + whole) * G + cta : s_cut[0] + walk) : walk * G + ((walk & 1) ? (G - 1 - cta) : cta);
    int j0 = 0;
    if constexpr (CUT) {
      if (walk == 0) j0 = s_cut[1];
      if (walk >= 0 && (w > s_cut[2] || (w == s_cut[2] && j0 >= s_cut[3]))) return false;
    }
    if (w >= n_items) return false;
    int pair;
    if (!CUT && causal) {
      const int rank = w / BH;
      it.bh = w - rank * BH;
      pair = n_pairs - 1 - rank;
    } else {  // equal weights: the pairs of a head run side by side and share its K / V in L2
      it.bh = w / n_pairs;
      pair = w - it.bh * n_pairs;
    }
    it.m0 = pair * (2 * BM);
    it.b = it.bh / a.H;
    it.h = it.bh - it.b * a.H;
    if (sorted) it.b = order[it.b], it.bh = it.b * a.H + it.h;
    it.n_valid = L;
    if (a.mask.kind == JVPFA_MASK_KVLEN) {
      const int n = a.mask.kv_len[it.b];
      it.n_valid = n < 0 ? 0 : (n > L ? L : n);
    }
    {
      int e0 = it.m0 < L ? it.n_valid : 0, e1 = it.m0 + BM < L ? it.n_valid : 0;
      if (causal) e0 = min(e0, it.m0 + BM), e1 = min(e1, it.m0 + 2 * BM);
      it.nt0 = (e0 + BN - 1) / BN, it.nt1 = (e1 + BN - 1) / BN;
      it.last0 = it.nt0 - 1, it.last1 = it.nt1 - 1;
      it.live0 = it.live1 = nullptr;
    }
    if constexpr (MK == 3) {
      // the bitmap has the mask's own extents: broadcast dimensions (stride 0) have one entry
      const int n_words = ((L + BN - 1) / BN + 63) >> 6;
      const long long hm = (a.mask.stride[0] ? (long long)it.b * (a.mask.stride[1] ? a.H : 1) : 0) +
                           (a.mask.stride[1] ? it.h : 0);
      auto scan = [&](int x, int& nt, int& last, const unsigned long long*& live) {
        const int qt = min(it.m0 / BM + x, n_q_tiles - 1);
        const long long qm = a.mask.stride[2] ? hm * n_q_tiles + qt : hm;
        live = reinterpret_cast<const unsigned long long*>(a.mask_tile_live) + qm * n_words;
        last = -1;
        for (int w2 = 0; w2 < (nt + 63) >> 6; ++w2) {
          unsigned long long bits = __ldg(live + w2);
          const int rem = nt - 64 * w2;
          if (rem < 64) bits &= (1ull << rem) - 1ull;
          if (bits) last = 64 * w2 + 63 - __clzll(bits);
        }
        if (last < 0) nt = 0;  // nothing to attend to: zeros and lse = +inf, as for kv_len = 0
      };
      scan(0, it.nt0, it.last0, it.live0);
      scan(1, it.nt1, it.last1, it.live1);
    }
    it.j0 = j0;
    it.n_load = max(it.nt0, it.nt1);
    if constexpr (CUT) {
      if (w == s_cut[2]) it.n_load = s_cut[3];
      it.last0 = min(it.nt0, it.n_load) - 1, it.last1 = min(it.nt1, it.n_load) - 1;
      if (it.last0 < j0) it.last0 = -1;
      if (it.last1 < j0) it.last1 = -1;
    }
    return true;
  };
  // This thread's place in the workspace for its row of query tile x of the item, which is cut; nullptr: it is not.
  auto share = [&](int walk, int x, int row) -> float4* {
    if (!CUT) return nullptr;
    const int place = walk < 0 ? -1 : cut_place(s_cut, s_cut[0] + walk, cta);
    return place < 0 ? nullptr
                     : reinterpret_cast<float4*>(shares + PairShare<DUAL>::HEAD / 4 + (size_t)place * PairShare<DUAL>::SIZE +
                                                 x * PairShare<DUAL>::TILE) + row;
  };

  // lse = NaN for every row of this CTA's items: the results of this launch are not to be trusted
  auto poison = [&]() {
    PairItem it;
    for (int walk = begin_items(); get_item(walk, it); ++walk) {
      const int i = it.m0 + tid;
      if (CUT && tid < 2 * BM) {
        float4* to = share(walk, tid / BM, tid % BM);
        if (to) to[PairShare<DUAL>::PIECES * BM] = make_float4(poison_f32(), poison_f32(), poison_f32(), 0.f);
      }
      if (tid < 2 * BM && i < L) a.lse[(size_t)it.bh * L + i] = poison_f32();
    }
  };
  if (dead_on_entry) {
    poison();
    return;
  }

  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(kv_full + s, 1);
      mbar_init(kv_empty + s, 2);
      if (BIAS) mbar_init(v_full + s, 1), mbar_init(v_empty + s, 2);
    }
    for (int x = 0; x < 2; ++x) {
      mbar_init(s_full + x, 1);
      mbar_init(s_free + x, 128);
      mbar_init(p_full + x, 128);
      mbar_init(pv_done + x, 1);
      mbar_init(o_free + x, 128);
      mbar_init(wg_bar + x, 128);
      if (BIAS) mbar_init(b_full + x, 1), mbar_init(b_empty + x, 128);
    }
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

  // Phase counters, kept alike by every role: g counts the key tiles loaded by this CTA (ring stage g % STAGES),
  // kact the items that load anything (q_full / q_empty), t[X] the key tiles query tile X has used (s_full,
  // s_free, p_full, pv_done of X complete once per such tile), kx[X] the items in which X used a tile (o_free).
  // The four warps of warpgroup 0 need few registers; the softmax threads hold two score tiles each.  (In the branches of the
  // roles: ptxas holds code behind a join of the two to the smaller number.)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0) {
        prefetch_tmap(&maps.q), prefetch_tmap(&maps.k), prefetch_tmap(&maps.v);
        if constexpr (DUAL) prefetch_tmap(&maps.tq), prefetch_tmap(&maps.tk), prefetch_tmap(&maps.tv);
        if constexpr (BIAS) prefetch_tmap(&maps.bias);
        int g = 0, kact = 0, nb0 = 0, nb1 = 0;  // nb: bias tiles of either query tile
        bool ok = true;
        PairItem it;
        for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
          if (it.n_load == 0) continue;
          // The Q tiles are single-buffered: both issuers must be through with the previous item's.
          if (kact > 0 && !mbar_wait(q_empty, (kact - 1) & 1, ab, kAbortQFull)) break;
          mbar_expect_tx(q_full, C::NQ * C::N_QT * C::Q_BYTES);
#pragma unroll
          for (int x = 0; x < 2; ++x) {  // a tile that starts past L reads as zeros
            unsigned char* dst = sQ + x * C::N_QT * C::Q_BYTES;
            tma_load_4d(dst, &maps.q, q_full, 0, it.m0 + x * BM, it.h, it.b);
            if constexpr (DUAL) tma_load_4d(dst + C::Q_BYTES, &maps.tq, q_full, 0, it.m0 + x * BM, it.h, it.b);
          }
          TileUse<MK> use(it);
          for (int j = it.j0; j < it.n_load; ++j) {
            const int m = use(j);
            if (m == 0) continue;
            const int st = g % STAGES, n0 = j * BN;
            const uint32_t free_par = ((g / STAGES) & 1) ^ 1;
            if (!mbar_wait(kv_empty + st, free_par, ab, kAbortKvEmpty)) {
              ok = false;
              break;
            }
            unsigned char *kd = sK + st * C::STAGE_BYTES, *vd = sV + st * C::STAGE_BYTES;
            mbar_expect_tx(kv_full + st, (BIAS ? 1 : 2) * C::HALF_BYTES);
            tma_load_4d(kd, &maps.k, kv_full + st, 0, n0, it.h, it.b);
            if constexpr (DUAL) tma_load_4d(kd + C::KV_BYTES, &maps.tk, kv_full + st, 0, n0, it.h, it.b);
            uint64_t* const vbar = BIAS ? v_full + st : kv_full + st;
            if constexpr (BIAS) {
              // one bias tile for each query tile that uses the key tile, when the one before has been added
              bool got = true;
              for (int x = 0; x < 2 && got; ++x) {
                if (!(m & (1 << x))) continue;
                int& nb = x ? nb1 : nb0;
                got = mbar_wait(b_empty + x, (nb & 1) ^ 1, ab, kAbortAux);
                if (!got) break;
                ++nb;
                mbar_expect_tx(b_full + x, C::B_BYTES);
                const int y = a.mask.stride[2] ? it.m0 + x * BM : 0, z = a.mask.stride[1] ? it.h : 0, w = a.mask.stride[0] ? it.b : 0;
                tma_load_4d(sB + x * C::B_BYTES, &maps.bias, b_full + x, n0, y, z, w);
                // Its place comes free a tile later, which is too late for DRAM: B2 H12 L2048 without tangents on a B200 77 -> 73.7 us.
                for (int n = j == it.j0 ? 1 : 2; n <= 2; ++n)
                  if (j + n < (x ? it.nt1 : it.nt0) && j + n < it.n_load) tma_prefetch_4d(&maps.bias, n0 + n * BN, y, z, w);
              }
              if (!got || !mbar_wait(v_empty + st, free_par, ab, kAbortKvEmpty)) {
                ok = false;
                break;
              }
              mbar_expect_tx(vbar, C::HALF_BYTES);
            }
            tma_load_4d(vd, &maps.v, vbar, 0, n0, it.h, it.b);
            if constexpr (DUAL) tma_load_4d(vd + C::KV_BYTES, &maps.tv, vbar, 0, n0, it.h, it.b);
            ++g;
          }
          ++kact;
        }
      }
    } else if (warp <= 2) {
      // ------------------------------------------------------------------ issuer of query tile X
      // A converged warp, one elected lane (mbar_wait_warp).  Whatever it executes between two MMAs is pure latency for the tensor
      // pipe, so stage and barrier cursors, parities and the low words of the operand descriptors live in registers and advance by
      // additions (descriptor = constant high word kDescHi + (byte address >> 4) in the low word).
      {
        const int X = warp - 1;
        constexpr uint32_t idesc_s = make_idesc(Fmt<T>::kIdesc, BM, BN, 0, 0);       // 128 x 64
        constexpr uint32_t idesc_s2 = make_idesc(Fmt<T>::kIdesc, BM, 2 * BN, 0, 0);  // 128 x 128: [S | tS]
        constexpr uint32_t idesc_o = make_idesc(Fmt<T>::kIdesc, BM, D, 0, 1);        // 128 x 64, B MN-major
        constexpr uint32_t idesc_o2 = make_idesc(Fmt<T>::kIdesc, BM, 2 * D, 0, 1);   // 128 x 128: [O | tO']
        constexpr uint32_t kLoV = (uint32_t)(C::KV_BYTES >> 4) << 16;  // [V | tV]: 64-column chunks KV_BYTES apart
        constexpr uint32_t STAGE16 = C::STAGE_BYTES >> 4;
        const uint32_t q_lo = kDescLo | (smem_u32(sQ + X * C::N_QT * C::Q_BYTES) >> 4), tq_lo = q_lo + (C::Q_BYTES >> 4);
        const uint32_t p_lo = kDescLo | (smem_u32(sP + X * C::N_P * C::P_BYTES) >> 4), w_lo = p_lo + (C::P_BYTES >> 4);
        const uint32_t k_lo0 = kDescLo | (smem_u32(sK) >> 4);
        const uint32_t v_lo0 = kLoV | (smem_u32(sV) >> 4);
        const uint32_t bar_kv_full = smem_u32(kv_full), bar_kv_empty = smem_u32(kv_empty);
        const uint32_t bar_v_full = smem_u32(v_full), bar_v_empty = smem_u32(BIAS ? v_empty : kv_empty);
        const uint32_t bar_s_full = smem_u32(s_full + X), bar_s_free = smem_u32(s_free + X);
        const uint32_t bar_p_full = smem_u32(p_full + X), bar_pv_done = smem_u32(pv_done + X);
        const uint32_t bar_o_free = smem_u32(o_free + X), bar_q_empty = smem_u32(q_empty);
        const uint32_t tq = tmem + X * C::COLS_PER_Q;
        uint32_t st = 0, st_par = 0;  // ring stage of the next loaded tile and the parity of its kv_full phase
        uint32_t tpar = 0;            // parity of the phase that this query tile's next used tile completes
        bool any_t = false;           // this query tile has used a tile before
        int kact = 0, kx = 0;
        bool ok = true;
        PairItem it;

        // [O | tO'] (+)= P [V | tV] ; tO' += W V for the tile in ring stage pst, whose phases have parity ppar (of V's stage: vpar)
        auto issue_pv = [&](uint32_t pst, uint32_t ppar, uint32_t vpar, bool first) -> bool {
          if (!mbar_wait_warp_u32(bar_p_full, ppar, ab, kAbortPFull)) return false;
          if (BIAS && !mbar_wait_warp_u32(bar_v_full + 8 * pst, vpar, ab, kAbortKvFull)) return false;
          // The item's first tile overwrites O / tO': the previous item's epilogue must have read them.
          if (first && kx > 0 && !mbar_wait_warp_u32(bar_o_free, (kx - 1) & 1, ab, kAbortOFull)) return false;
          tc_fence_after();
          const uint32_t v_lo = v_lo0 + pst * STAGE16;
          if (elect_one()) {
            if constexpr (DUAL) {
              umma_ss_lo_dyn(tq + C::COL_O, p_lo, v_lo, idesc_o2, first ? 0u : 1u);
#pragma unroll
              for (int kk = 1; kk < BN / 16; ++kk) umma_ss_lo<true>(tq + C::COL_O, p_lo + kk * 2, v_lo + kk * 128, idesc_o2);
#pragma unroll
              for (int kk = 0; kk < BN / 16; ++kk) umma_ss_lo<true>(tq + C::COL_TO, w_lo + kk * 2, v_lo + kk * 128, idesc_o);
            } else {  // P from TMEM
              umma_ts_lo_dyn(tq + C::COL_O, tq + C::COL_P, v_lo, idesc_o, first ? 0u : 1u);
#pragma unroll
              for (int kk = 1; kk < BN / 16; ++kk) umma_ts_lo<true>(tq + C::COL_O, tq + C::COL_P + kk * 8, v_lo + kk * 128, idesc_o);
            }
            tc_commit_u32(bar_v_empty + 8 * pst);
            tc_commit_u32(bar_pv_done);
          }
          return true;
        };

        for (int walk = begin_items(); ok && get_item(walk, it); ++walk) {
          if (it.n_load == 0) continue;
          // waited for by both issuers in every item, used or not: a parity wait must see every phase
          if (!mbar_wait_warp(q_full, kact & 1, ab, kAbortQFull)) break;
          const int my_last = it.last(X);
          bool pend = false, pend_first = false, first = true;
          uint32_t pend_st = 0, pend_par = 0, pend_vpar = 0;
          TileUse<MK> use(it);
          for (int j = it.j0; j < it.n_load; ++j) {
            const int m = use(j);
            if (m == 0) continue;
            if (!mbar_wait_warp_u32(bar_kv_full + 8 * st, st_par, ab, kAbortKvFull)) {
              ok = false;
              break;
            }
            if (m & (1 << X)) {
              // S / tS of the previous tile (of this item or the one before) must be in the softmax threads' registers
              if (any_t && !mbar_wait_warp_u32(bar_s_free, tpar ^ 1, ab, kAbortSFull)) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint32_t k_lo = k_lo0 + st * STAGE16;
              if (elect_one()) {
                if constexpr (DUAL) {
                  umma_ss_lo<false>(tq + C::COL_S, q_lo, k_lo, idesc_s2);  // [S | tS] = Q [K ; tK]^T
#pragma unroll
                  for (int ks = 1; ks < D / 16; ++ks)
                    if (ks < 2 || a.D > 32) umma_ss_lo<true>(tq + C::COL_S, q_lo + ks * 2, k_lo + ks * 2, idesc_s2);
#pragma unroll
                  for (int ks = 0; ks < D / 16; ++ks)
                    if (ks < 2 || a.D > 32) umma_ss_lo<true>(tq + C::COL_TS, tq_lo + ks * 2, k_lo + ks * 2, idesc_s);  // tS += tQ K^T
                } else {
                  umma_ss_lo<false>(tq + C::COL_S, q_lo, k_lo, idesc_s);
#pragma unroll
                  for (int ks = 1; ks < D / 16; ++ks)
                    if (ks < 2 || a.D > 32) umma_ss_lo<true>(tq + C::COL_S, q_lo + ks * 2, k_lo + ks * 2, idesc_s);
                }
                tc_commit_u32(bar_s_full);
                if constexpr (BIAS) tc_commit_u32(bar_kv_empty + 8 * st);
                if (j == my_last) tc_commit_u32(bar_q_empty);  // arrives when the item's last scores are complete
              }
              if (pend && !issue_pv(pend_st, pend_par, pend_vpar, pend_first)) {
                ok = false;
                break;
              }
              pend = true, pend_st = st, pend_par = tpar, pend_vpar = st_par, pend_first = first, first = false;
              tpar ^= 1, any_t = true;
            } else {
              // Loaded for the other query tile only.  A pending output product holds an older ring stage: it goes
              // out first, or the producer could wait for that stage while this thread waits for the producer.
              if (pend) {
                if (!issue_pv(pend_st, pend_par, pend_vpar, pend_first)) {
                  ok = false;
                  break;
                }
                pend = false;
              }
              if (BIAS && !mbar_wait_warp_u32(bar_v_full + 8 * st, st_par, ab, kAbortKvFull)) {  // (its stage's turn, not an earlier one)
                ok = false;
                break;
              }
              if (elect_one()) {
                mbar_arrive(kv_empty + st);
                if (BIAS) mbar_arrive(v_empty + st);
              }
            }
            if (++st == STAGES) st = 0, st_par ^= 1;
          }
          if (!ok) break;
          if (pend && !issue_pv(pend_st, pend_par, pend_vpar, pend_first)) break;
          if (!first)
            ++kx;  // this query tile used key tiles in the item (its q_empty arrival went out with the last scores)
          else if (elect_one())
            mbar_arrive(q_empty);
          ++kact;
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ------------------------------------------------------------------ softmax + epilogue of query tile X
    const int X = (warp - 4) >> 2;
    const int quarter = warp & 3;  // the TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t tq = tmem + lane_off + X * C::COLS_PER_Q;
    const uint32_t tS = tq + C::COL_S, tTS = tq + C::COL_TS, tO = tq + C::COL_O, tTO = tq + C::COL_TO;
    // this thread's row of the P / W tiles: 16-byte chunk c sits at position c ^ (row & 7) of the 128-byte row
    const uint32_t pP = smem_u32(sP + X * C::N_P * C::P_BYTES) + row * 128, pW = pP + C::P_BYTES;
    const uint32_t sw = (uint32_t)(row & 7);
    const float scale_log2 = a.sm_scale * kLog2e;
    const float2 c2 = make_float2(scale_log2, scale_log2);
    const float2 sc2 = make_float2(a.sm_scale, a.sm_scale);
    bool alive = true;
    uint32_t t = 0;

    // The item's O / tO rows leave through the query tile's P / W buffers (idle between items) and one TMA store
    // per output, issued by the warpgroup's first thread.  Before anybody writes those buffers again the store
    // must have read them: release_staging().
    bool store_pending = false;
    uint32_t wg_phase = 0;
    auto wg_sync = [&]() -> bool {
      mbar_arrive(wg_bar + X);
      const bool ok = mbar_wait(wg_bar + X, wg_phase & 1, ab, kAbortAux);
      ++wg_phase;
      return ok;
    };
    auto release_staging = [&]() -> bool {
      if (!store_pending) return true;
      store_pending = false;
      if (row == 0) tma_store_wait_read();
      return wg_sync();
    };
    // Normalise and store one item's rows.  has_acc: the accumulators hold something (the query tile used key
    // tiles); then the last tile's output MMAs are waited for and O / tO' are released afterwards.
    auto epilogue = [&](const PairItem& it, int i, float m_used, float l_run, float mu_run, bool has_acc) -> bool {
      if (has_acc) {
        if (!mbar_wait(pv_done + X, (t - 1) & 1, ab, kAbortOFull)) return false;
        tc_fence_after();
      }
      if (!release_staging()) return false;
      const bool empty = !(l_run > 0.f);
      const float inv_l = empty ? 0.f : 1.f / l_run;
      const float mu_n = mu_run * inv_l;
      if (i < L) {
        a.lse[(size_t)it.bh * L + i] = empty ? INFINITY : (m_used + log2f(l_run));
        if constexpr (DUAL) a.mu[(size_t)it.bh * L + i] = mu_n;
      }
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t ro[32], rt[DUAL ? 32 : 1];
        uint32_t po[16];
        if (has_acc) {
          tmem_ld32(tO + 32 * c, ro);
          if constexpr (DUAL) tmem_ld32(tTO + 32 * c, rt);
          tmem_wait_ld();
          if (c == D / 32 - 1) {  // everything is in registers: the accumulators may be overwritten
            tc_fence_before();
            mbar_arrive(o_free + X);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            ro[e] = 0u;
            if constexpr (DUAL) rt[e] = 0u;
          }
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) ro[e] = __float_as_uint(__uint_as_float(ro[e]) * inv_l);
#pragma unroll
        for (int e = 0; e < 16; ++e) po[e] = Elem<T>::pack(__uint_as_float(ro[2 * e]), __uint_as_float(ro[2 * e + 1]));
#pragma unroll
        for (int e = 0; e < 4; ++e)
          st_shared_v4(pP + (((uint32_t)(4 * c + e) ^ sw) << 4), po[4 * e], po[4 * e + 1], po[4 * e + 2], po[4 * e + 3]);
        if constexpr (DUAL) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float t0 = __uint_as_float(rt[2 * e]) * inv_l - mu_n * __uint_as_float(ro[2 * e]);
            const float t1 = __uint_as_float(rt[2 * e + 1]) * inv_l - mu_n * __uint_as_float(ro[2 * e + 1]);
            po[e] = Elem<T>::pack(t0, t1);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            st_shared_v4(pW + (((uint32_t)(4 * c + e) ^ sw) << 4), po[4 * e], po[4 * e + 1], po[4 * e + 2], po[4 * e + 3]);
        }
      }
      fence_proxy_async_smem();
      if (!wg_sync()) return false;
      const int mX = it.m0 + X * BM;
      if (row == 0 && mX < L) {
        tma_store_4d(&maps.o, sP + X * C::N_P * C::P_BYTES, 0, mX, it.h, it.b);
        if constexpr (DUAL) tma_store_4d(&maps.to, sP + X * C::N_P * C::P_BYTES + C::P_BYTES, 0, mX, it.h, it.b);
        tma_store_commit();
      }
      store_pending = true;
      return true;
    };

    // What this CTA has of a row of a pair that is cut.
    auto store_share = [&](float4* to, float m_used, float l_run, float mu_run) -> bool {
      if (!mbar_wait(pv_done + X, (t - 1) & 1, ab, kAbortOFull)) return false;
      tc_fence_after();
      to[PairShare<DUAL>::PIECES * BM] = make_float4(m_used, l_run, mu_run, 0.f);
#pragma unroll 1
      for (int c = 0; c < PairShare<DUAL>::PIECES; c += 8) {
        uint32_t r[32];
        tmem_ld32(tO + 4 * c, r);  // (tO' follows O)
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e)
          reinterpret_cast<uint4*>(to)[(c + e) * BM] = make_uint4(r[4 * e], r[4 * e + 1], r[4 * e + 2], r[4 * e + 3]);
      }
      tc_fence_before();
      mbar_arrive(o_free + X);
      return true;
    };

    PairItem it;
    for (int walk = begin_items(); alive && get_item(walk, it); ++walk) {
      const int mX = it.m0 + X * BM;
      const int i = mX + row;
      const bool used = !CUT || it.last(X) >= 0;
      if (it.last(X) < 0) {  // no live key for this query tile: zeros, lse = +inf
        if constexpr (!CUT) {
          alive = epilogue(it, i, -INFINITY, 0.f, 0.f, false);
          continue;
        } else if (float4* const to = share(walk, X, row)) {
          to[PairShare<DUAL>::PIECES * BM] = make_float4(-INFINITY, 0.f, 0.f, 1.f);
          continue;
        }
      }
      const float slack = a.flags & kExactRowMax ? 0.f : 8.f;
      float m_used = -INFINITY, l_run = 0.f, mu_run = 0.f;
      // MK != 0: this thread's row of the mask / bias (rows past L are clamped; their results are not stored)
      constexpr bool BOOLM = MK == 1 || MK == 3;
      const unsigned char* mrow = nullptr;
      const uint32_t* brow = nullptr;  // packed boolean mask
      if constexpr (BOOLM) {
        if (a.mask_bits != nullptr)
          brow = mask_bit_row(a.mask_bits, a.mask, mask_head(a.mask, it.b, it.h, a.H), min(i, L - 1), L);
      }
      if constexpr (BOOLM)
        mrow = reinterpret_cast<const unsigned char*>(a.mask.ptr) + (long long)it.b * a.mask.stride[0] + (long long)it.h * a.mask.stride[1] +
               (long long)min(i, L - 1) * a.mask.stride[2];
      // The mask's piece of a tile.  Where the next tile is known it is requested as soon as this one's has been
      // used: at its own tile's beginning the scores are there already, and the loads would be waited for.  (Without a condition,
      // zeros beyond the last tile: else this tile's piece would have to be kept.)
      uint2 next_keys = make_uint2(~0u, ~0u);
      auto fetch_mask = [&](int n0) {
        if constexpr (BOOLM) {
          if (brow != nullptr) {
            next_keys = n0 < L ? ldg_nc_v2(brow + (n0 >> 5)) : make_uint2(0u, 0u);
          } else {
            next_keys.x = mask_piece_bits(mrow + n0, n0, L) | mask_piece_bits(mrow + n0 + 16, n0 + 16, L) << 16;
            next_keys.y = mask_piece_bits(mrow + n0 + 32, n0 + 32, L) | mask_piece_bits(mrow + n0 + 48, n0 + 48, L) << 16;
          }
        }
      };
      constexpr bool AHEAD = MK == 1;
      if constexpr (AHEAD) fetch_mask(it.j0 * BN);
      TileUse<MK> use(it);
      bool first = true;  // the item's first tile used by this query tile
      uint32_t s_ok = 0u;
      for (int j = it.j0; j < it.n_load; ++j) {
        if (!(use(j) & (1 << X))) continue;
        const int n0 = j * BN;
        if constexpr (MK == 3) fetch_mask(n0);
        uint2 keys = next_keys;  // BOOLM: bit c of (x, y) = the mask lets this row attend key n0 + c
        if (!s_ok && !mbar_wait(s_full + X, t & 1, ab, kAbortSFull)) {
          alive = false;
          break;
        }
        tc_fence_after();
        uint32_t x0[32], x1[32];
        tmem_ld32(tS, x0);
        tmem_ld32(tS + 32, x1);
        tmem_wait_ld();
        if constexpr (!DUAL) {  // (the tangent scores follow half a tile at a time, when their probabilities are formed)
          tc_fence_before();
          mbar_arrive(s_free + X);
        }
        // live key columns of this row inside the tile: col < col_hi
        int col_hi = min(BN, it.n_valid - n0);
        if (causal) col_hi = min(col_hi, i - n0 + 1);
        const bool partial = (n0 + BN > it.n_valid) || (causal && n0 + BN - 1 > mX);
        // Row maximum of the tile in log2 units.  Without a bias it is taken over the raw scores (the scale is
        // positive) and the scaling is folded into the exponent's multiply-add; otherwise the scores are scaled,
        // biased and masked first.
        float mx;
        if constexpr (BOOLM) {
          if (partial) keys.x &= first_columns(col_hi), keys.y &= first_columns(col_hi - 32);
          if (__any_sync(0xffffffffu, (keys.x & keys.y) != ~0u)) {  // (inside a window or a document no entry is False)
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (!((keys.x >> c) & 1u)) x0[c] = 0xff800000u;  // -inf
              if (!((keys.y >> c) & 1u)) x1[c] = 0xff800000u;
            }
          }
        }
        if constexpr (MK != 2) {
          if (MK == 0 && partial) {
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              if (c >= col_hi) x0[c] = 0xff800000u;  // -inf
              if (32 + c >= col_hi) x1[c] = 0xff800000u;
            }
          }
          float mxa = -INFINITY, mxb = -INFINITY, mxc = -INFINITY, mxd = -INFINITY;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            mxa = max3(mxa, __uint_as_float(x0[4 * c]), __uint_as_float(x0[4 * c + 1]));
            mxb = max3(mxb, __uint_as_float(x0[4 * c + 2]), __uint_as_float(x0[4 * c + 3]));
            mxc = max3(mxc, __uint_as_float(x1[4 * c]), __uint_as_float(x1[4 * c + 1]));
            mxd = max3(mxd, __uint_as_float(x1[4 * c + 2]), __uint_as_float(x1[4 * c + 3]));
          }
          mx = max3(mxa, mxb, fmaxf(mxc, mxd)) * scale_log2;
        } else {
          if (!mbar_wait(b_full + X, t & 1, ab, kAbortAux)) {
            alive = false;
            break;
          }
          // this row of the tile (a bias of one row: the first): 16-byte piece c sits at position c ^ (row & 7)
          const uint32_t brow_sm = smem_u32(sB + X * C::B_BYTES) + (a.mask.stride[2] ? row * 128 : 0), bsw = a.mask.stride[2] ? sw : 0u;
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w0[4], w1[4];
            lds_v4(brow_sm + (((uint32_t)q ^ bsw) << 4), w0);
            lds_v4(brow_sm + (((uint32_t)(4 + q) ^ bsw) << 4), w1);
            if (q == 3) mbar_arrive_behind(b_empty + X, w1[3], opaque_zero(a));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int c = 4 * q + e;
              // scores are in log2 units: bias * log2(e)
              const float2 l2 = make_float2(kLog2e, kLog2e);
              float2 v0 = __ffma2_rn(unpack2<T>(w0[e]), l2, __fmul2_rn(pf2(x0[2 * c], x0[2 * c + 1]), c2));
              float2 v1 = __ffma2_rn(unpack2<T>(w1[e]), l2, __fmul2_rn(pf2(x1[2 * c], x1[2 * c + 1]), c2));
              if (partial) {
                if (2 * c >= col_hi) v0.x = -INFINITY;
                if (2 * c + 1 >= col_hi) v0.y = -INFINITY;
                if (32 + 2 * c >= col_hi) v1.x = -INFINITY;
                if (33 + 2 * c >= col_hi) v1.y = -INFINITY;
              }
              x0[2 * c] = __float_as_uint(v0.x), x0[2 * c + 1] = __float_as_uint(v0.y);
              x1[2 * c] = __float_as_uint(v1.x), x1[2 * c + 1] = __float_as_uint(v1.y);
              mx0 = fmaxf(mx0, v0.x), mx1 = fmaxf(mx1, v0.y), mx2 = fmaxf(mx2, v1.x), mx3 = fmaxf(mx3, v1.y);
            }
          }
          mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        }
        if constexpr (MK == 1) fetch_mask(n0 + BN);
        // Lazy running max: keep the old reference while the new maximum is at most 2^8 above it (kExactRowMax: never).
        const bool grow = mx > m_used + slack;
        float alpha = 1.f;
        if (grow) {
          alpha = fast_exp2(m_used - mx);
          m_used = mx;
        }
        const float m_eff = (m_used == -INFINITY) ? 0.f : m_used;
        bool prev_pv_seen = false;  // the previous tile's output MMAs are known to be complete
        if (!first && __any_sync(0xffffffffu, grow)) {
          // O / tO' are rescaled in place: the previous tile's output MMAs must have landed
          if (!mbar_wait(pv_done + X, (t - 1) & 1, ab, kAbortOFull)) {
            alive = false;
            break;
          }
          prev_pv_seen = true;
          tc_fence_after();
          const float2 al2 = make_float2(alpha, alpha);
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            // Head dimension 32: the second half holds zeros.  (Its reference is the exact maximum, so most tiles come here: with tangents B3 H13
            // L3296 315 -> 298 us, B4 H8 L1000 35.1 -> 34.1.)
            if (32 * c >= a.D) break;
            uint32_t r[32];
            tmem_ld32(tO + 32 * c, r);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const float2 v = __fmul2_rn(pf2(r[2 * e], r[2 * e + 1]), al2);
              r[2 * e] = __float_as_uint(v.x), r[2 * e + 1] = __float_as_uint(v.y);
            }
            tmem_st32(tO + 32 * c, r);
            if constexpr (DUAL) {
              tmem_ld32(tTO + 32 * c, r);
              tmem_wait_ld();
#pragma unroll
              for (int e = 0; e < 16; ++e) {
                const float2 v = __fmul2_rn(pf2(r[2 * e], r[2 * e + 1]), al2);
                r[2 * e] = __float_as_uint(v.x), r[2 * e + 1] = __float_as_uint(v.y);
              }
              tmem_st32(tTO + 32 * c, r);
            }
          }
          tmem_wait_st();
        }
        // Exponentials, row sums, W = P * tS * scale and the packing to 16 bit in one loop per half tile, so that
        // the special-function unit's latency is covered by the arithmetic of the neighbouring columns.
        // The P / W tiles are single-buffered: the previous tile's output MMAs must have read them.  (A look at the barrier takes 100
        // cycles and more also when they are long complete: it is taken under the first half's arithmetic.)
        const uint32_t pv_ok = t == 0 || prev_pv_seen ? 1u : mbar_test_quiet(pv_done + X, (t - 1) & 1);
        uint32_t ts0[DUAL ? 32 : 1], ts1[DUAL ? 32 : 1];
        if constexpr (DUAL) {
          tmem_ld32(tTS, ts0);
          tmem_ld32(tTS + 32, ts1);
          tmem_wait_ld();
          tc_fence_before();
          mbar_arrive(s_free + X);  // both score accumulators are in registers now
        }
        const float2 nm2 = make_float2(-m_eff, -m_eff);
        float2 ls2 = make_float2(0.f, 0.f), ms2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t* xs = hh ? x1 : x0;
          uint32_t pp[16], wp[DUAL ? 16 : 1];
          const uint32_t* ts = hh ? ts1 : ts0;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float2 e;
            if constexpr (MK != 2)
              e = __ffma2_rn(pf2(xs[2 * c], xs[2 * c + 1]), c2, nm2);
            else
              e = __fadd2_rn(pf2(xs[2 * c], xs[2 * c + 1]), nm2);
            const float2 pv = make_float2(fast_exp2(e.x), fast_exp2(e.y));
            ls2 = __fadd2_rn(ls2, pv);
            pp[c] = Elem<T>::pack(pv.x, pv.y);
            if constexpr (DUAL) {
              const float2 w = __fmul2_rn(pv, __fmul2_rn(pf2(ts[2 * c], ts[2 * c + 1]), sc2));
              ms2 = __fadd2_rn(ms2, w);
              wp[c] = Elem<T>::pack(w.x, w.y);
            }
          }
          if (hh == 0 && ((!pv_ok && !mbar_wait(pv_done + X, (t - 1) & 1, ab, kAbortOFull)) ||
                          (first && !release_staging()))) {  // (the previous item's output store has read the buffers)
            alive = false;
            break;
          }
          if constexpr (DUAL) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {  // chunk 4 hh + c = key columns 8 (4 hh + c) ..
              const uint32_t off = ((uint32_t)(4 * hh + c) ^ sw) << 4;
              st_shared_v4(pP + off, pp[4 * c], pp[4 * c + 1], pp[4 * c + 2], pp[4 * c + 3]);
              st_shared_v4(pW + off, wp[4 * c], wp[4 * c + 1], wp[4 * c + 2], wp[4 * c + 3]);
            }
          } else {
            if (hh == 0) tc_fence_after();  // (behind the look or the wait: the stores follow what pv_done says has been read)
            tmem_st16(tq + C::COL_P + 16 * hh, pp);
          }
        }
        if (!alive) break;

        l_run = l_run * alpha + (ls2.x + ls2.y);
        if constexpr (DUAL) mu_run = mu_run * alpha + (ms2.x + ms2.y);
        if constexpr (DUAL) {
          fence_proxy_async_smem();
        } else {
          s_ok = mbar_test_quiet(s_full + X, (t + 1) & 1);  // (of the next tile, under the stores' way: 117 -> 115 us at H64 L2048)
          tmem_wait_st();
        }
        tc_fence_before();
        mbar_arrive(p_full + X);
        first = false;
        ++t;
      }
      if (!alive) break;
      if (float4* const to = share(walk, X, row)) {
        if (!store_share(to, m_used, l_run, mu_run)) break;
      } else {
        if (!epilogue(it, i, m_used, l_run, mu_run, used)) break;
      }
    }
    if (row == 0) tma_store_wait_all();  // shared memory must outlive the stores that read it
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

// The rows of the pairs that were cut.  Block x of 8 * (ctas - 1) looks at where CTA x / 8 + 1 begins; a pair that is cut there first is
// this block's, an eighth of it: 128 rows of one query tile, 8 columns a thread of O and, at the same places, of tO.  Bound by reading
// the shares: B2 H12 L2048 with tangents, 44 pairs among 148 CTAs, has 168 of 135 KB, 22.7 MB (11.8 us).  A pair has two shares at least,
// and two are requested before the first is looked at; those beyond (one or two there) are read one after another.
template <typename T, bool DUAL>
__global__ void __launch_bounds__(256) pair64_finish_kernel(const jvpfa_fwd_args a, const float* shares, int ctas) {
  using S = PairShare<DUAL>;
  behind_previous();
  const int2* begin = reinterpret_cast<const int2*>(shares);
  const int j = blockIdx.x / 8 + 1;
  const int2 first = begin[j], before = begin[j - 1];
  int2 next = j + 1 < ctas ? begin[j + 1] : make_int2(-1, 0);
  if (first.y == 0 || (before.x == first.x && before.y > 0)) return;
  const int x = (blockIdx.x >> 2) & 1, row = threadIdx.x & 127, piece = 4 * (blockIdx.x & 3) + 2 * (threadIdx.x >> 7);
  const float4* base = reinterpret_cast<const float4*>(shares + S::HEAD / 4) + x * (S::TILE / 4) + row;
  struct Share {
    float4 st, o[2], to[DUAL ? 2 : 1];
  };
  auto load = [&](int place, Share& v) {
    const float4* p = base + (size_t)place * (S::SIZE / 4);
    v.st = p[S::PIECES * 128];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v.o[h] = p[(piece + h) * 128];
      if constexpr (DUAL) v.to[h] = p[(16 + piece + h) * 128];
    }
  };
  float m = -INFINITY, l = 0.f, mu = 0.f, o[8] = {}, to[8] = {};
  bool gave_up = false;
  auto add = [&](const Share& v) {
    if (v.st.w != 0.f) return;  // no key of the share, and nothing but its statistics is there
    // As in the loop over key tiles, the reference is 0 where the maximum is -inf: maxima pass over what is not a number, so a share of
    // such a maximum may have sums that are none.
    const float top = fmaxf(m, v.st.x), ref = top == -INFINITY ? 0.f : top, keep = fast_exp2(m - ref), w = fast_exp2(v.st.x - ref);
    gave_up = gave_up || isnan(v.st.x);  // (a CTA that gave up wrote it: no maximum is NaN)
    m = top;
    l = keep * l + w * v.st.y;
    mu = keep * mu + w * v.st.z;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      o[4 * h] = keep * o[4 * h] + w * v.o[h].x, o[4 * h + 1] = keep * o[4 * h + 1] + w * v.o[h].y;
      o[4 * h + 2] = keep * o[4 * h + 2] + w * v.o[h].z, o[4 * h + 3] = keep * o[4 * h + 3] + w * v.o[h].w;
      if constexpr (DUAL) {
        to[4 * h] = keep * to[4 * h] + w * v.to[h].x, to[4 * h + 1] = keep * to[4 * h + 1] + w * v.to[h].y;
        to[4 * h + 2] = keep * to[4 * h + 2] + w * v.to[h].z, to[4 * h + 3] = keep * to[4 * h + 3] + w * v.to[h].w;
      }
    }
  };
  Share u, v;
  load(2 * (j - 1) + 1, u);  // the share that begins the pair is its CTA's last
  v.st.w = 1.f;
  if (next.x != first.x || next.y != first.y) load(2 * j, v);  // (else CTA j has nothing to do)
  add(u);
  add(v);
  int2 cur = next;
  for (int c = j + 1; cur.x == first.x && cur.y > 0; ++c) {
    next = c + 1 < ctas ? begin[c + 1] : make_int2(-1, 0);
    if (next.x != cur.x || next.y != cur.y) {
      load(2 * c, u);
      add(u);
    }
    cur = next;
  }
  const int item = first.x;
  const int n_pairs = (a.L + 255) / 256, bh = item / n_pairs, i = (item - bh * n_pairs) * 256 + x * 128 + row;
  if (i >= a.L) return;
  const bool empty = !(l > 0.f);
  const float inv_l = empty ? 0.f : 1.f / l, mu_n = mu * inv_l;
  const size_t at = (size_t)bh * a.L + i;
  if (piece == 0) {
    a.lse[at] = gave_up ? poison_f32() : empty ? INFINITY : m + log2f(l);
    if constexpr (DUAL) a.mu[at] = mu_n;
  }
  if (4 * piece >= a.D) return;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    o[e] *= inv_l;
    if constexpr (DUAL) to[e] = to[e] * inv_l - mu_n * o[e];
  }
  auto store = [&](void* p, const float (&v)[8]) {
    *reinterpret_cast<uint4*>(static_cast<T*>(p) + at * a.D + 4 * piece) =
        make_uint4(Elem<T>::pack(v[0], v[1]), Elem<T>::pack(v[2], v[3]), Elem<T>::pack(v[4], v[5]), Elem<T>::pack(v[6], v[7]));
  };
  store(a.o, o);
  if constexpr (DUAL) store(a.to, to);
}

static int pair_sm_count() {
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

// How the pairs are dealt: `ctas` CTAs among which their key tiles are shared out, after `whole` rounds of pairs as a whole; ctas = 0: all
// as a whole.  Both ways in key tiles of the CTA that has the most.  The shares' way through the workspace takes as long as 8, 9 behind whole
// rounds, and 12 where most CTAs have two of them; a twentieth less is asked for.  Measured on a B200, replayed from a graph, us whole /
// shared out, bf16 with tangents: H4 L1024 27 / 20, H16 L1024 27 / 26, H24 L1024 31 / 35 (left whole), H48 L1024 52 / 47, H4 L2048 46 / 28, H24
// L2048 91 / 74, H30 L2048 91 / 90 and with a bias 123 / 125, H12 L4096 169 / 129; causal H16 L1024 25 / 23, H24 L2048 52 / 55
// (left whole), H8 L4096 86 / 59; without tangents H4 L1024 19 / 14, H24 L1024 21 / 23 (left whole).
// Where tiles are stepped over their numbers are not known here: whole.
// Key padding: whole where the lengths are not known here either.  With them the way of the shares counts as one more (pieces end anywhere in
// ragged entries, so more pairs are cut).  Without tangents, lengths of about L / 10 and L / 2, whole / shared out as if there were no padding: B2 H12
// L2048 13.2 / 19.3 and 29.3 / 31.2, B8 H2 L1024 7.6 / 13.0 and 12.7 / 16.3 (left whole), H4 L4096 12.0 / 15.8 (left whole) and 35.9 / 26.1.
struct PairDeal {
  int ctas, whole;
};
static PairDeal deal_pairs(const jvpfa_fwd_args& a, int sms) {
  constexpr PairDeal all_whole{0, 0};
  if (a.mask.kind == JVPFA_MASK_BOOL && a.mask_tile_live != nullptr) return all_whole;
  const bool causal = a.mask.kind == JVPFA_MASK_CAUSAL, keys = a.mask.kind == JVPFA_MASK_KVLEN;
  if (keys && a.kv_len_host == nullptr) return all_whole;
  const long long P = (a.L + 255) / 256, N = (a.L + 63) / 64, BH = (long long)a.B * a.H, items = P * BH;
  const long long line = BH * (causal ? P * (P + 1) * 2 : P * N) + items * kPairOpen;  // (of keys: at most)
  const long long G = items < sms ? items : sms;
  const HostLengths lengths(a.kv_len_host, a.B, a.L, keys && a.B <= kMaxSortedBatch && items > G);
  long long steps = BH * (causal ? (P - 1) * P * 2 + N : P * N);
  if (keys) {
    steps = 0;
    for (int b = 0; b < a.B; ++b) steps += lengths.tiles(b, 64) * a.H * P;
  }
  const long long ctas = steps / 4 < sms ? steps / 4 : sms;
  if (ctas < 2 || !cut_fits(line, ctas)) return all_whole;
  const long long rounds = (items + G - 1) / G;
  if (rounds > (causal ? 8 : keys ? 16 : rounds)) return all_whole;  // (the lightest are dealt last and even out)
  const long long most = causal ? most_loaded(items, G, 8, [&](long long w) { return N < 4 * (P - w / BH) ? N : 4 * (P - w / BH); })
                         : keys ? most_loaded(items, G, 16, [&](long long w) { return lengths.tiles(w / (a.H * P), 64); })
                                : rounds * N;
  const long long whole = causal || keys ? 0 : items / ctas;
  const long long shared = whole > 0 ? whole * N + (items - whole * ctas) * N / ctas + 9 : steps / ctas + (2 * items > ctas ? 12 : 8) + keys;
  return shared * 20 < most * 19 ? PairDeal{(int)ctas, (int)whole} : all_whole;
}

template <typename T, bool DUAL, int MK, bool CUT>
static cudaError_t run_pair64(const jvpfa_fwd_args& a, const FwdPairMaps& maps, float* shares, int whole, int* status, int grid, cudaStream_t stream) {
  using C = FwdPairCfg<DUAL, MK == 2>;
  auto kern = fwd_tc5_pair64_kernel<T, DUAL, MK, CUT>;
  static SmemOptIn opt_in;
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), C::SMEM_BYTES)) return cudaErrorInvalidValue;
  return launch_behind(kern, grid, C::NTHREADS, C::SMEM_BYTES, stream, a, maps, shares, whole, status);
}

template <typename T, bool DUAL, int MK>
static int launch_pair64(const jvpfa_fwd_args& a, cudaStream_t stream) {
  using C = FwdPairCfg<DUAL, MK == 2>;
  int* status = tc5_status_device_ptr();
  if (!status) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  FwdPairMaps maps;
  const long long BH = (long long)a.B * a.H;
  const CUtensorMapDataType dt = Fmt<T>::kTma;
  // (64, L, H, B) maps: the inputs may be strided views (in_stride), e.g. (B,L,H,D) tensors seen as (B,H,L,D)
  const int64_t* st = a.in_stride;
  bool ok = encode_map4d(&maps.q, dt, a.q, a.D, a.L, a.H, a.B, st, C::BM) && encode_map4d(&maps.k, dt, a.k, a.D, a.L, a.H, a.B, st, C::BN) &&
            encode_map4d(&maps.v, dt, a.v, a.D, a.L, a.H, a.B, st, C::BN);
  if (DUAL)
    ok = ok && encode_map4d(&maps.tq, dt, a.tq, a.D, a.L, a.H, a.B, st, C::BM) &&
         encode_map4d(&maps.tk, dt, a.tk, a.D, a.L, a.H, a.B, st, C::BN) && encode_map4d(&maps.tv, dt, a.tv, a.D, a.L, a.H, a.B, st, C::BN);
  else
    maps.tq = maps.tk = maps.tv = maps.q;
  ok = ok && encode_map4d(&maps.o, dt, a.o, a.D, a.L, a.H, a.B, nullptr, C::BM);
  if (DUAL)
    ok = ok && encode_map4d(&maps.to, dt, a.to, a.D, a.L, a.H, a.B, nullptr, C::BM);
  else
    maps.to = maps.o;
  maps.bias = maps.q;
  if (MK == 2) ok = ok && encode_map_bias(&maps.bias, dt, a.mask, a.L, a.H, a.B, C::BM);
  if (!ok) {
    set_last_cuda_error(cudaErrorUnknown, "cuTensorMapEncodeTiled(fwd pair64)");
    return JVPFA_ERR_CUDA;
  }
  const int sms = pair_sm_count();
  if (sms <= 0) {
    set_last_cuda_error(cudaErrorUnknown, "multiprocessor count");
    return JVPFA_ERR_CUDA;
  }
  const long long n_q_tiles = (a.L + C::BM - 1) / C::BM;
  const long long n_items = ((n_q_tiles + 1) / 2) * BH;
  const int grid = (int)(n_items < sms ? n_items : sms);
  cudaError_t e;
  if constexpr (MK != 3) {
    const auto [ctas, whole] = deal_pairs(a, sms);
    if (ctas > 0 && a.workspace != nullptr && (reinterpret_cast<uintptr_t>(a.workspace) & 15u) == 0 &&
        a.workspace_bytes >= PairShare<DUAL>::bytes(ctas)) {
      float* shares = static_cast<float*>(a.workspace);
      e = run_pair64<T, DUAL, MK, true>(a, maps, shares, whole, status, ctas, stream);
      if (e == cudaSuccess) {
        e = launch_behind(pair64_finish_kernel<T, DUAL>, 8 * (ctas - 1), 256, 0, stream, a, static_cast<const float*>(shares), ctas);
      }
    } else {
      e = run_pair64<T, DUAL, MK, false>(a, maps, nullptr, 0, status, grid, stream);
    }
  } else {
    e = run_pair64<T, DUAL, MK, false>(a, maps, nullptr, 0, status, grid, stream);
  }
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch fwd_tc5_pair64");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <typename T>
static int launch_pair64_t(const jvpfa_fwd_args& a, cudaStream_t s) {
  const bool dual = a.tq != nullptr;
  if (a.mask.kind == JVPFA_MASK_BOOL && a.mask_tile_live != nullptr)
    return dual ? launch_pair64<T, true, 3>(a, s) : launch_pair64<T, false, 3>(a, s);
  if (a.mask.kind == JVPFA_MASK_BOOL) return dual ? launch_pair64<T, true, 1>(a, s) : launch_pair64<T, false, 1>(a, s);
  if (a.mask.kind == JVPFA_MASK_BIAS) return dual ? launch_pair64<T, true, 2>(a, s) : launch_pair64<T, false, 2>(a, s);
  return dual ? launch_pair64<T, true, 0>(a, s) : launch_pair64<T, false, 0>(a, s);
}

}  // namespace tc5

// What the launch can use where pairs are cut.
long long fwd_pair64_workspace(const jvpfa_fwd_args& a) {
  if (a.impl == JVPFA_IMPL_GENERIC || a.D > 64 || !fwd_tc5_eligible(a)) return 0;
  const int ctas = tc5::deal_pairs(a, tc5::pair_sm_count()).ctas;
  return ctas == 0 ? 0 : a.tq != nullptr ? tc5::PairShare<true>::bytes(ctas) : tc5::PairShare<false>::bytes(ctas);
}

int launch_fwd_tc5_pair64(const jvpfa_fwd_args& a, cudaStream_t s) {
  return a.dtype == JVPFA_BF16 ? tc5::launch_pair64_t<__nv_bfloat16>(a, s) : tc5::launch_pair64_t<__half>(a, s);
}

}  // namespace jvpfa
