// Backward for fp32 tensors on pairs of fp16 numbers (fp32_split.cuh).  Math and structure as in bwd_generic.cu: one kernel
// owns key tiles and loops over queries (dK, dV), one owns query tiles and loops over keys (dQ); a warp takes 16 owned rows
// and 16 rows of every loop tile, and the partial sums of the KG warps of a row group are added once at the end (in a fixed
// order: results stay reproducible bit for bit).
//
// Bound like the forward (fwd_fp32.cu) by latency: dK and dV together take the registers that two outputs take there.
// B200, B2 H8 L1024 D128, against three TF32 products split in every warp: dQ through tO with bias 798 -> 438 us, through O
// 440 -> 230 us; B2 H4 L256 D64, both outputs: dK and dV 27.6 -> 21.4 us, dQ 22.5 -> 18.3 us.  Error against 64 bits: 3e-7 to
// 1.2e-6 (TF32 pairs: 6e-7 to 4.3e-6).
#include "fp32_split.cuh"

namespace jvpfa {

namespace {

using namespace f32;

// RESIDENT: CTAs on an SM.  Two where shared memory allows and there are enough of them (64-row tiles): they wait at
// different times, which is worth more than what D = 64 and 128 then spill (B2 H8 L1024 D64: dQ through both outputs 272 ->
// 245 us, dK and dV 348 -> 306 us; L500, with 96 tiles: 57 -> 72 us, so not there).  Otherwise two stages where there is room.
template <int D, int OWN_TILES, int LOOP_TILES, int RG, int KG, bool STATS, int RESIDENT>
struct BwdCfg {
  static constexpr int kResident = RESIDENT;
  static constexpr int OWN = 16 * RG, LOOP = 16 * KG, NT = 32 * RG * KG;
  static constexpr int kOwn = OWN * D * 4, kLoop = LOOP * D * 4;  // bytes of a tile
  static constexpr int STAGES = OWN_TILES * kOwn + 2 * LOOP_TILES * kLoop <= 200 * 1024 / RESIDENT ? 2 : 1;
  static constexpr int kMerge = RG * KG / 2 * 16 * D * 4;  // reuses the ring
  static constexpr int kRing = STAGES * LOOP_TILES * kLoop > kMerge ? STAGES * LOOP_TILES * kLoop : kMerge;
  static constexpr int NSTAT = 5;  // lse, delta, eps, cterm, mu of the loop's queries
  static constexpr int kFloats = OWN_TILES * OWN + STAGES * LOOP_TILES * LOOP + (STATS ? STAGES * NSTAT * LOOP : 0);
  static constexpr size_t smem = (size_t)OWN_TILES * kOwn + kRing + 4 * kFloats;
};

struct HeadView {  // where this CTA's head lies
  size_t off, stat;
  long long in_off, in_rs;
  __device__ HeadView(const jvpfa_bwd_args& a, int bh, int b, int h, int D) {
    off = (size_t)bh * a.L * D;
    stat = (size_t)bh * a.L;
    const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
    in_off = strided ? (long long)b * a.in_stride[0] + (long long)h * a.in_stride[1] : (long long)off;
    in_rs = strided ? a.in_stride[2] : D;
  }
  __device__ const float* in(const void* p) const { return reinterpret_cast<const float*>(p) + in_off; }
  __device__ const float* dense(const void* p) const { return reinterpret_cast<const float*>(p) + off; }
};

// TKV: K and V have tangents (JVPFA_ZERO_TKV leaves out what they would be multiplied by).
// ---- dK, dV.  Tiles are held transposed (rows = keys, columns = queries), so that P^T etc. feed the second products from
// registers. ----
template <int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG>
using DkdvCfg = BwdCfg<D, TKV ? 4 : 2, 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0), RG, KG, true, RG == 4 && D <= 64 ? 2 : 1>;

template <int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG>
__global__ void __launch_bounds__(32 * RG * KG, DkdvCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>::kResident) bwd_dkdv_fp32_kernel(const jvpfa_bwd_args a) {
  using C = DkdvCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  constexpr int BN = C::OWN, BM = C::LOOP, NT = C::NT, STAGES = C::STAGES, ND = D / 8;
  constexpr int OWN_TILES = TKV ? 4 : 2, LOOP_TILES = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0);
  constexpr int kGO = 1, kTQ = 1 + (HAS_GO ? 1 : 0), kG = kTQ + 1;  // loop tiles after Q

  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sOwn = smem_raw;  // K, V, tK, tV
  unsigned char* sLoop = sOwn + OWN_TILES * C::kOwn;
  float* iOwn = reinterpret_cast<float*>(sLoop + C::kRing);
  float* iLoop = iOwn + OWN_TILES * BN;
  float* sStat = iLoop + STAGES * LOOP_TILES * BM;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y, b = bh / a.H, h = bh - b * a.H;
  const int n0 = blockIdx.x * BN;
  const HeadView hv(a, bh, b, h, D);
  const MaskView mv = make_mask_view(a.mask, b, h, L);

  // query tiles that can see this key tile
  int m_begin = 0;
  if (mv.kind == JVPFA_MASK_CAUSAL) m_begin = (n0 / BM) * BM;
  int n_tiles = (L - m_begin + BM - 1) / BM;
  if (mv.kind == JVPFA_MASK_KVLEN && n0 >= mv.kv_len) n_tiles = 0;

  auto copy_loop = [&](int it) {
    const int stage = it & (STAGES - 1), m0 = m_begin + it * BM;
    unsigned char* base = sLoop + stage * LOOP_TILES * C::kLoop;
    copy_tile<BM, D, NT>(base, hv.in(a.q), m0, L, tid, hv.in_rs);
    if constexpr (HAS_GO) copy_tile<BM, D, NT>(base + kGO * C::kLoop, hv.dense(a.go), m0, L, tid, D);
    if constexpr (HAS_GT) {
      copy_tile<BM, D, NT>(base + kTQ * C::kLoop, hv.in(a.tq), m0, L, tid, hv.in_rs);
      copy_tile<BM, D, NT>(base + kG * C::kLoop, hv.dense(a.gto), m0, L, tid, D);
    }
    cp_async_commit();
    if (tid < BM) {
      float* st = sStat + stage * C::NSTAT * BM + tid;
      const int i = m0 + tid;
      const bool ok = i < L;
      st[0] = ok ? a.lse[hv.stat + i] : INFINITY;
      st[BM] = ok ? a.delta[hv.stat + i] : 0.f;
      if constexpr (HAS_GT) {
        st[2 * BM] = ok ? a.eps[hv.stat + i] : 0.f;
        st[3 * BM] = ok ? a.cterm[hv.stat + i] : 0.f;
        st[4 * BM] = ok ? a.mu[hv.stat + i] : 0.f;
      }
    }
  };
  auto split_loop = [&](int it) {
    const int stage = it & (STAGES - 1);
    split_tiles<LOOP_TILES * BM, BM, D, NT>(sLoop + stage * LOOP_TILES * C::kLoop, iLoop + stage * LOOP_TILES * BM, tid);
  };

  copy_tile<BN, D, NT>(sOwn, hv.in(a.k), n0, L, tid, hv.in_rs);
  copy_tile<BN, D, NT>(sOwn + C::kOwn, hv.in(a.v), n0, L, tid, hv.in_rs);
  if constexpr (TKV) {
    copy_tile<BN, D, NT>(sOwn + 2 * C::kOwn, hv.in(a.tk), n0, L, tid, hv.in_rs);
    copy_tile<BN, D, NT>(sOwn + 3 * C::kOwn, hv.in(a.tv), n0, L, tid, hv.in_rs);
  }
  if (n_tiles > 0) copy_loop(0);
  cp_async_commit();
  cp_async_wait<0>();
  split_tiles<OWN_TILES * BN, BN, D, NT>(sOwn, iOwn, tid);
  if (n_tiles > 0) split_loop(0);
  if (STAGES == 2 && n_tiles > 1) copy_loop(1);
  __syncthreads();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16, qr = kg * 16;
  const int key_lo = n0 + r0 + g, key_hi = key_lo + 8;
  const uint32_t aK = smem_addr(sOwn), aV = aK + C::kOwn, aTK = aK + 2 * C::kOwn, aTV = aK + 3 * C::kOwn;

  float dk[ND][4], dv[ND][4];
  zero<ND>(dk);
  zero<ND>(dv);

  for (int it = 0; it < n_tiles; ++it) {
    // this warp's queries of the tile (none of them may see its keys: nothing to do)
    const int mw = m_begin + it * BM + qr;
    if (mw < L && !(mv.kind == JVPFA_MASK_CAUSAL && mw + 16 <= n0 + r0)) {
      const int stage = it & (STAGES - 1);
      const uint32_t aQ = smem_addr(sLoop + stage * LOOP_TILES * C::kLoop);
      const uint32_t aGO = aQ + kGO * C::kLoop, aTQ = aQ + kTQ * C::kLoop, aG = aQ + kG * C::kLoop;
      const float* iq = iLoop + stage * LOOP_TILES * BM + qr;
      const float *igo = iq + kGO * BM, *itq = iq + kTQ * BM, *ig = iq + kG * BM;
      const float* st = sStat + stage * C::NSTAT * BM + qr;

      bool ok[2][4];  // fetched ahead of the products that hide its latency
      float bias[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = mw + n * 8 + 2 * t + (e & 1), j = (e < 2) ? key_lo : key_hi;
          ok[n][e] = mv.allowed(i, j);
          bias[n][e] = ok[n][e] ? mv.bias(i, j) : 0.f;
        }
      }
      // P^T, A^T = P*(tS - mu), gtS^T, gS^T
      float p[2][4], ts[2][4], e_[2][4], f[2][4];
      {
        float y2[2][4];
        scores<D, TKV, HAS_GT, C::kResident == 1>(p, ts, y2, aK, aTK, aQ, aTQ, r0, qr, lane);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float ik = iOwn[r0 + g + 8 * r], itk = TKV ? iOwn[2 * BN + r0 + g + 8 * r] : 0.f;
#pragma unroll
          for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int e = 2 * r + c, j = n * 8 + 2 * t + c;
              const float s = p[n][e] * ik * iq[j];
              p[n][e] = ok[n][e] ? exp2f(s * scale_log2 + bias[n][e] * kLog2e - st[j]) : 0.f;
              if constexpr (TKV)
                ts[n][e] = fmaf(ts[n][e] * itk, iq[j], y2[n][e] * ik * itq[j]) * a.sm_scale;
              else if constexpr (HAS_GT)
                ts[n][e] = y2[n][e] * ik * itq[j] * a.sm_scale;
            }
          }
        }
      }
      {
        float y1[2][4], y2[2][4];
        if constexpr (HAS_GT)
          scores<D, TKV, HAS_GO, C::kResident == 1>(e_, y1, y2, aV, aTV, aG, aGO, r0, qr, lane);
        else
          scores<D, false, false, C::kResident == 1>(y2, y1, y1, aV, aV, aGO, aGO, r0, qr, lane);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float iv = iOwn[BN + r0 + g + 8 * r], itv = TKV ? iOwn[3 * BN + r0 + g + 8 * r] : 0.f;
#pragma unroll
          for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int e = 2 * r + c, j = n * 8 + 2 * t + c;
              const float pv = p[n][e];
              float x = HAS_GO ? y2[n][e] * iv * igo[j] : 0.f, sub = st[BM + j];
              if constexpr (HAS_GT) {
                const float tsv = ts[n][e], ev = e_[n][e] * iv * ig[j], eps = st[2 * BM + j], mu = st[4 * BM + j];
                if constexpr (TKV) x = fmaf(y1[n][e] * itv, ig[j], x);
                sub += st[3 * BM + j];
                x += ev * (tsv - mu) - eps * tsv;
                e_[n][e] = pv * (ev - eps);  // gtS
                ts[n][e] = pv * (tsv - mu);  // A
              }
              f[n][e] = pv * (x - sub);  // gS
            }
          }
        }
      }
      // dV += P^T gO + A^T G;  dK += gS^T Q + gtS^T tQ
      PairA f0, f1;
      float k0[2], k1[2];
      if constexpr (HAS_GO) a_from_acc(f0, k0, p, igo, lane);
      if constexpr (HAS_GT) a_from_acc(f1, k1, ts, ig, lane);
      outputs<D, HAS_GO, HAS_GT>(dv, f0, k0, f1, k1, aGO, aG, qr, lane);
      a_from_acc(f0, k0, f, iq, lane);
      if constexpr (HAS_GT) a_from_acc(f1, k1, e_, itq, lane);
      outputs<D, true, HAS_GT>(dk, f0, k0, f1, k1, aQ, aTQ, qr, lane);
    }
    if (it + 1 < n_tiles) {
      if constexpr (STAGES == 1) {
        __syncthreads();  // every warp is done with the only stage
        copy_loop(it + 1);
      }
      cp_async_wait<0>();
      split_loop(it + 1);
      __syncthreads();  // the next tile is there, and every warp is done with this one
      if (STAGES == 2 && it + 2 < n_tiles) copy_loop(it + 2);
    }
  }
  __syncthreads();
  merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dk, rg, kg, lane);
  merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dv, rg, kg, lane);
  if (kg != 0) return;
  const float fk[2] = {a.sm_scale, a.sm_scale}, fv[2] = {1.f, 1.f};
  store_strip<D>(reinterpret_cast<float*>(a.dk) + hv.off, dk, fk, key_lo, L, lane);
  store_strip<D>(reinterpret_cast<float*>(a.dv) + hv.off, dv, fv, key_lo, L, lane);
}

// ---- dQ (rows = queries, columns = keys) ----
template <int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG>
using DqCfg = BwdCfg<D, 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0), TKV ? 4 : 2, RG, KG, false,
                     RG == 4 && (D <= 64 || !HAS_GT) ? 2 : 1>;

template <int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG>
__global__ void __launch_bounds__(32 * RG * KG, DqCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>::kResident) bwd_dq_fp32_kernel(const jvpfa_bwd_args a) {
  using C = DqCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  constexpr int BM = C::OWN, BN = C::LOOP, NT = C::NT, STAGES = C::STAGES, ND = D / 8;
  constexpr int OWN_TILES = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0), LOOP_TILES = TKV ? 4 : 2;
  constexpr int kGO = 1, kTQ = 1 + (HAS_GO ? 1 : 0), kG = kTQ + 1;  // own tiles after Q

  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sOwn = smem_raw;
  unsigned char* sLoop = sOwn + OWN_TILES * C::kOwn;  // K, V, tK, tV
  float* iOwn = reinterpret_cast<float*>(sLoop + C::kRing);
  float* iLoop = iOwn + OWN_TILES * BM;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y, b = bh / a.H, h = bh - b * a.H;
  const int m0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * BM;  // heaviest causal tiles first
  const HeadView hv(a, bh, b, h, D);
  const MaskView mv = make_mask_view(a.mask, b, h, L);

  int n_end = L;
  if (mv.kind == JVPFA_MASK_CAUSAL) n_end = min(L, m0 + BM);
  if (mv.kind == JVPFA_MASK_KVLEN) n_end = min(L, mv.kv_len);
  const int n_tiles = (n_end + BN - 1) / BN;

  auto copy_loop = [&](int it) {
    unsigned char* base = sLoop + (it & (STAGES - 1)) * LOOP_TILES * C::kLoop;
    copy_tile<BN, D, NT>(base, hv.in(a.k), it * BN, L, tid, hv.in_rs);
    copy_tile<BN, D, NT>(base + C::kLoop, hv.in(a.v), it * BN, L, tid, hv.in_rs);
    if constexpr (TKV) {
      copy_tile<BN, D, NT>(base + 2 * C::kLoop, hv.in(a.tk), it * BN, L, tid, hv.in_rs);
      copy_tile<BN, D, NT>(base + 3 * C::kLoop, hv.in(a.tv), it * BN, L, tid, hv.in_rs);
    }
    cp_async_commit();
  };
  auto split_loop = [&](int it) {
    const int stage = it & (STAGES - 1);
    split_tiles<LOOP_TILES * BN, BN, D, NT>(sLoop + stage * LOOP_TILES * C::kLoop, iLoop + stage * LOOP_TILES * BN, tid);
  };

  copy_tile<BM, D, NT>(sOwn, hv.in(a.q), m0, L, tid, hv.in_rs);
  if constexpr (HAS_GO) copy_tile<BM, D, NT>(sOwn + kGO * C::kOwn, hv.dense(a.go), m0, L, tid, D);
  if constexpr (HAS_GT) {
    copy_tile<BM, D, NT>(sOwn + kTQ * C::kOwn, hv.in(a.tq), m0, L, tid, hv.in_rs);
    copy_tile<BM, D, NT>(sOwn + kG * C::kOwn, hv.dense(a.gto), m0, L, tid, D);
  }
  if (n_tiles > 0) copy_loop(0);
  cp_async_commit();
  cp_async_wait<0>();
  split_tiles<OWN_TILES * BM, BM, D, NT>(sOwn, iOwn, tid);
  if (n_tiles > 0) split_loop(0);
  if (STAGES == 2 && n_tiles > 1) copy_loop(1);
  __syncthreads();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16, kr = kg * 16;
  // D = 128 with two CTAs on an SM: the addresses of fully unrolled products are what spills (432 -> 64 bytes; 242 -> 223 us at
  // B2 H8 L1024 through O).  Elsewhere the loop costs more than it saves (D = 64, same shape: 114 -> 122 us).
  constexpr int kUnroll = D == 128 && C::kResident == 2 ? 2 : D / 16;
  const int row_lo = m0 + r0 + g;
  const uint32_t aQ = smem_addr(sOwn), aGO = aQ + kGO * C::kOwn, aTQ = aQ + kTQ * C::kOwn, aG = aQ + kG * C::kOwn;
  float lse[2], sub[2], eps[2] = {0.f, 0.f}, mu[2] = {0.f, 0.f};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = row_lo + 8 * r;
    const bool ok = row < L;
    lse[r] = ok ? a.lse[hv.stat + row] : INFINITY;
    sub[r] = ok ? a.delta[hv.stat + row] : 0.f;
    if constexpr (HAS_GT) {
      sub[r] += ok ? a.cterm[hv.stat + row] : 0.f;
      eps[r] = ok ? a.eps[hv.stat + row] : 0.f;
      mu[r] = ok ? a.mu[hv.stat + row] : 0.f;
    }
  }

  float dq[ND][4];
  zero<ND>(dq);

  for (int it = 0; it < n_tiles; ++it) {
    const int nw = it * BN + kr;  // this warp's keys of the tile
    if (nw < n_end && !(mv.kind == JVPFA_MASK_CAUSAL && nw > m0 + r0 + 15)) {
      const int stage = it & (STAGES - 1);
      const uint32_t aK = smem_addr(sLoop + stage * LOOP_TILES * C::kLoop), aV = aK + C::kLoop, aTK = aK + 2 * C::kLoop,
                     aTV = aK + 3 * C::kLoop;
      const float* ik = iLoop + stage * LOOP_TILES * BN + kr;
      const float *iv = ik + BN, *itk = ik + 2 * BN, *itv = ik + 3 * BN;

      bool ok[2][4];  // fetched ahead of the products that hide its latency
      float bias[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mv.pair(row_lo, nw + n * 8 + 2 * t, &ok[n][0], &bias[n][0]);
        mv.pair(row_lo + 8, nw + n * 8 + 2 * t, &ok[n][2], &bias[n][2]);
      }
      float p[2][4], ts[2][4], e_[2][4], f[2][4];
      {
        float y2[2][4];
        scores<D, HAS_GT, TKV, C::kResident == 1, kUnroll>(p, ts, y2, aQ, aTQ, aK, aTK, r0, kr, lane);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float iq = iOwn[r0 + g + 8 * r], itq = HAS_GT ? iOwn[kTQ * BM + r0 + g + 8 * r] : 0.f;
#pragma unroll
          for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int e = 2 * r + c, j = n * 8 + 2 * t + c;
              const float s = p[n][e] * iq * ik[j];
              p[n][e] = ok[n][e] ? exp2f(s * scale_log2 + bias[n][e] * kLog2e - lse[r]) : 0.f;
              if constexpr (TKV)
                ts[n][e] = fmaf(ts[n][e] * itq, ik[j], y2[n][e] * iq * itk[j]) * a.sm_scale;
              else if constexpr (HAS_GT)
                ts[n][e] = ts[n][e] * itq * ik[j] * a.sm_scale;
            }
          }
        }
      }
      {
        // E = G V^T, dP = gO V^T, F = G tV^T
        float y1[2][4], y2[2][4];
        if constexpr (HAS_GT)
          scores<D, HAS_GO, TKV, C::kResident == 1, kUnroll>(e_, y1, y2, aG, aGO, aV, aTV, r0, kr, lane);
        else
          scores<D, false, false, C::kResident == 1, kUnroll>(y1, y2, y2, aGO, aGO, aV, aV, r0, kr, lane);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float igo = HAS_GO ? iOwn[kGO * BM + r0 + g + 8 * r] : 0.f, ig = HAS_GT ? iOwn[kG * BM + r0 + g + 8 * r] : 0.f;
#pragma unroll
          for (int n = 0; n < 2; ++n) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const int e = 2 * r + c, j = n * 8 + 2 * t + c;
              const float pv = p[n][e];
              float x = HAS_GO ? y1[n][e] * igo * iv[j] : 0.f;
              if constexpr (HAS_GT) {
                const float tsv = ts[n][e], ev = e_[n][e] * ig * iv[j];
                if constexpr (TKV) x = fmaf(y2[n][e] * ig, itv[j], x);
                x += ev * (tsv - mu[r]) - eps[r] * tsv;
                e_[n][e] = pv * (ev - eps[r]);  // gtS
              }
              f[n][e] = pv * (x - sub[r]);  // gS
            }
          }
        }
      }
      PairA f0, f1;  // gS K + gtS tK
      float k0[2], k1[2];
      a_from_acc(f0, k0, f, ik, lane);
      if constexpr (TKV) a_from_acc(f1, k1, e_, itk, lane);
      outputs<D, true, TKV>(dq, f0, k0, f1, k1, aK, aTK, kr, lane);
    }
    if (it + 1 < n_tiles) {
      if constexpr (STAGES == 1) {
        __syncthreads();  // every warp is done with the only stage
        copy_loop(it + 1);
      }
      cp_async_wait<0>();
      split_loop(it + 1);
      __syncthreads();  // the next tile is there, and every warp is done with this one
      if (STAGES == 2 && it + 2 < n_tiles) copy_loop(it + 2);
    }
  }
  __syncthreads();
  merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dq, rg, kg, lane);
  if (kg != 0) return;
  const float fq[2] = {a.sm_scale, a.sm_scale};
  store_strip<D>(reinterpret_cast<float*>(a.dq) + hv.off, dq, fq, row_lo, L, lane);
}

template <int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG>
int launch_one(const jvpfa_bwd_args& a, cudaStream_t stream) {
  using C1 = DkdvCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  using C2 = DqCfg<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  static_assert(C1::smem <= 227 * 1024 && C2::smem <= 227 * 1024, "shared memory of one CTA");
  auto k1 = bwd_dkdv_fp32_kernel<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  auto k2 = bwd_dq_fp32_kernel<D, HAS_GO, HAS_GT, TKV, RG, KG>;
  static SmemOptIn opt_in1, opt_in2;
  if (!opt_in1.ensure(reinterpret_cast<const void*>(k1), C1::smem) || !opt_in2.ensure(reinterpret_cast<const void*>(k2), C2::smem))
    return JVPFA_ERR_CUDA;
  const dim3 grid((a.L + C1::OWN - 1) / C1::OWN, a.B * a.H);
  if (!(a.flags & JVPFA_SKIP_DKDV)) k1<<<grid, C1::NT, C1::smem, stream>>>(a);
  if (!(a.flags & JVPFA_SKIP_DQ)) k2<<<grid, C2::NT, C2::smem, stream>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch bwd_fp32");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <int D>
int launch_d(const jvpfa_bwd_args& a, cudaStream_t s) {
  return dispatch_split<D>(a.B, a.H, a.L, [&](auto rg, auto kg) {
    constexpr int RG = decltype(rg)::value, KG = decltype(kg)::value;
    if (!a.gto) return launch_one<D, true, false, false, RG, KG>(a, s);
    if (a.flags & JVPFA_ZERO_TKV) return launch_one<D, false, true, false, RG, KG>(a, s);  // (go is refused with it)
    return a.go ? launch_one<D, true, true, true, RG, KG>(a, s) : launch_one<D, false, true, true, RG, KG>(a, s);
  });
}

}  // namespace

int launch_bwd_fp32(const jvpfa_bwd_args& a, cudaStream_t s) {
  switch (a.D) {
    case 32:
      return launch_d<32>(a, s);
    case 64:
      return launch_d<64>(a, s);
    case 128:
      return launch_d<128>(a, s);
    default:
      return JVPFA_ERR_SHAPE;
  }
}

}  // namespace jvpfa
