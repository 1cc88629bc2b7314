// Fused primal (+ tangent) attention forward for fp32 tensors on pairs of fp16 numbers (fp32_split.cuh).
//
// A CTA of RG x KG warps owns 16*RG query rows of one (batch, head).  Warp (rg, kg) owns 16 of the rows and 16 rows of every
// key tile; it keeps a running maximum, denominator, mu and output of its own over its keys, and the KG partial results of a
// row are merged once, through shared memory, when the keys are through.  While a tile is worked on, the next one arrives
// by cp.async; every thread splits what it copied itself, so a tile costs one barrier.
//
// Math as in fwd_generic.cu (S, tS, online softmax with mu = sum P*tS, O = P V, tO' = (P*tS) V + P tV).  Each of the three
// score products has its own accumulator, since each has its own pair of row scales.
//
// What bounds it: latency.  mma.sync multiplies 1024 fp16 pairs per clock and SM, of which it does some 45 %; the
// accumulators of two outputs at D = 128 leave room for two warps on each quarter of an SM, which wait for ldmatrix, for the
// softmax between the two sets of products and, once per tile, for the split.  Fetching the operands of the next step ahead
// of a step's products, both outputs in one sweep over V and four pieces of the split at a time took 466 to 402 us.
// B200, B2 H8 L1024 D128 with bias, against three TF32 products split in every warp: both outputs 683 -> 402 us, O alone 315
// -> 187 us; B2 H4 L256 D64, both outputs: 18.0 -> 16.7 us.  Error against 64 bits, over lengths 36 to 1410, all masks and
// head dimensions: 1e-7 to 7e-7 (O) and 2e-7 to 9e-7 (tO); TF32 pairs: 2e-7 to 1.2e-6 and 5e-7 to 2.3e-6.
#include "fp32_split.cuh"

namespace jvpfa {

namespace {

using namespace f32;

// TKV: K and V have tangents (JVPFA_ZERO_TKV leaves them, and two of the six products, out: B2 H8 L1024 D128 with bias 402
// -> 301 us, the backward through tO for dQ 438 -> 267 us).
template <int D, bool DUAL, bool TKV, int RG, int KG>
struct FwdCfg {
  static constexpr int BM = 16 * RG, BN = 16 * KG, NT = 32 * RG * KG;
  static constexpr int NQ = DUAL ? 2 : 1, NKV = TKV ? 4 : 2;
  static constexpr int kTile = BN * D * 4;
  // Two CTAs on an SM where registers allow (one output to accumulate, or a head dimension of 32) and there are enough of
  // them (64-row tiles): they wait at different times.  B2 H8 L2048: one output, D 64, 404 -> 316 us; both, D 32, 548 -> 437
  // us, but D 64 837 -> 861 us with what then spills.  Otherwise two stages where there is room.
  static constexpr int kResident = RG == 4 && (!DUAL || D == 32) ? 2 : 1;
  static constexpr int STAGES = 2 * NKV * kTile + NQ * BM * D * 4 <= 200 * 1024 / kResident ? 2 : 1;
  static constexpr int kMerge = KG > 1 ? RG * KG / 2 * 16 * D * 4 : 0;  // reuses the ring
  static constexpr int kRing = STAGES * NKV * kTile > kMerge ? STAGES * NKV * kTile : kMerge;
  static constexpr int kScales = NQ * BM + STAGES * NKV * BN, kRow = 3 * KG * BM;
  static constexpr size_t smem = (size_t)NQ * BM * D * 4 + kRing + 4 * (kScales + kRow);
};

template <int D, bool DUAL, bool TKV, int RG, int KG>
__global__ void __launch_bounds__(32 * RG * KG, FwdCfg<D, DUAL, TKV, RG, KG>::kResident) fwd_fp32_kernel(const jvpfa_fwd_args a) {
  using C = FwdCfg<D, DUAL, TKV, RG, KG>;
  constexpr int BM = C::BM, BN = C::BN, NT = C::NT, STAGES = C::STAGES, NKV = C::NKV, ND = D / 8;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* sQ = smem_raw;
  unsigned char* sTQ = sQ + BM * D * 4;  // DUAL
  unsigned char* sKV = sQ + C::NQ * BM * D * 4;
  float* iQ = reinterpret_cast<float*>(sKV + C::kRing);  // [NQ][BM]
  float* iKV = iQ + C::NQ * BM;                          // [STAGES][NKV][BN]
  float* sRow = iKV + STAGES * NKV * BN;                 // [3][KG][BM]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  const int m0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * BM;  // heaviest causal tiles first

  const size_t head_off = (size_t)bh * L * D;
  const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
  const long long in_off = strided ? (long long)b * a.in_stride[0] + (long long)h * a.in_stride[1] : (long long)head_off;
  const long long in_rs = strided ? a.in_stride[2] : D;
  auto head = [&](const void* p) { return reinterpret_cast<const float*>(p) + in_off; };

  const MaskView mv = make_mask_view(a.mask, b, h, L);
  int n_end = L;
  if (mv.kind == JVPFA_MASK_CAUSAL) n_end = min(L, m0 + BM);
  if (mv.kind == JVPFA_MASK_KVLEN) n_end = min(L, mv.kv_len);
  const int n_tiles = (n_end + BN - 1) / BN;

  auto copy_kv = [&](int it) {
    unsigned char* base = sKV + (it & (STAGES - 1)) * NKV * C::kTile;
    copy_tile<BN, D, NT>(base, head(a.k), it * BN, L, tid, in_rs);
    copy_tile<BN, D, NT>(base + C::kTile, head(a.v), it * BN, L, tid, in_rs);
    if constexpr (TKV) {
      copy_tile<BN, D, NT>(base + 2 * C::kTile, head(a.tk), it * BN, L, tid, in_rs);
      copy_tile<BN, D, NT>(base + 3 * C::kTile, head(a.tv), it * BN, L, tid, in_rs);
    }
    cp_async_commit();
  };
  auto split_kv = [&](int it) {
    const int stage = it & (STAGES - 1);
    split_tiles<NKV * BN, BN, D, NT>(sKV + stage * NKV * C::kTile, iKV + stage * NKV * BN, tid);
  };

  copy_tile<BM, D, NT>(sQ, head(a.q), m0, L, tid, in_rs);
  if constexpr (DUAL) copy_tile<BM, D, NT>(sTQ, head(a.tq), m0, L, tid, in_rs);
  if (n_tiles > 0) copy_kv(0);
  cp_async_commit();
  cp_async_wait<0>();
  split_tiles<C::NQ * BM, BM, D, NT>(sQ, iQ, tid);
  if (n_tiles > 0) split_kv(0);
  if (STAGES == 2 && n_tiles > 1) copy_kv(1);
  __syncthreads();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16;
  const int row_lo = m0 + r0 + g, row_hi = row_lo + 8;
  const uint32_t aQ = smem_addr(sQ), aTQ = smem_addr(sTQ);

  float acc_o[ND][4], acc_t[DUAL ? ND : 1][4];
  zero<ND>(acc_o);
  zero<DUAL ? ND : 1>(acc_t);
  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f}, mu_run[2] = {0.f, 0.f};

  for (int it = 0; it < n_tiles; ++it) {
    const int n0 = it * BN + kg * 16;  // this warp's keys of the tile
    // (a part beyond the end, or above the diagonal of the warp's rows, is nobody's work; the barrier below is everybody's)
    if (n0 < n_end && !(mv.kind == JVPFA_MASK_CAUSAL && n0 > m0 + r0 + 15)) {
      const int stage = it & (STAGES - 1), kr = kg * 16;
      const uint32_t aK = smem_addr(sKV + stage * NKV * C::kTile), aV = aK + C::kTile, aTK = aK + 2 * C::kTile, aTV = aK + 3 * C::kTile;
      const float* ik = iKV + stage * NKV * BN + kr;
      const float *iv = ik + BN, *itk = ik + 2 * BN, *itv = ik + 3 * BN;

      // user mask: fetched ahead of the products that hide its latency
      const bool full_tile = (mv.kind == JVPFA_MASK_NONE && n0 + 16 <= L && m0 + BM <= L) ||
                             (mv.kind == JVPFA_MASK_CAUSAL && n0 + 15 <= m0 + r0 && m0 + BM <= L) ||
                             (mv.kind == JVPFA_MASK_KVLEN && n0 + 16 <= mv.kv_len && m0 + BM <= L);
      bool ok[2][4];
      float bias[2][4];
      if (!full_tile) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          mv.pair(row_lo, n0 + n * 8 + 2 * t, &ok[n][0], &bias[n][0]);
          mv.pair(row_hi, n0 + n * 8 + 2 * t, &ok[n][2], &bias[n][2]);
        }
      }

      float s[2][4], y1[2][4], y2[2][4];
      scores<D, DUAL, TKV, C::kResident == 1>(s, y1, y2, aQ, aTQ, aK, aTK, r0, kr, lane);

      // take the scales back, mask / bias, move to the base-2 domain
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float iq = iQ[r0 + g + 8 * r], itq = DUAL ? iQ[BM + r0 + g + 8 * r] : 0.f;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int e = 2 * r + c, j = n * 8 + 2 * t + c;
            float x = s[n][e] * iq * ik[j] * scale_log2;
            if constexpr (TKV)
              y1[n][e] = fmaf(y1[n][e] * itq, ik[j], y2[n][e] * iq * itk[j]);
            else if constexpr (DUAL)
              y1[n][e] *= itq * ik[j];
            if (!full_tile) {
              if (ok[n][e]) {
                x += bias[n][e] * kLog2e;
              } else {
                x = -INFINITY;
                if constexpr (DUAL) y1[n][e] = 0.f;
              }
            }
            s[n][e] = x;
            mx[r] = fmaxf(mx[r], x);
          }
        }
      }
      float alpha[2], m_use[2], ls[2] = {0.f, 0.f}, ms[2] = {0.f, 0.f};
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float m_new = fmaxf(m_run[r], quad_max(mx[r]));
        m_use[r] = (m_new == -INFINITY) ? 0.f : m_new;
        alpha[r] = exp2f(m_run[r] - m_use[r]);  // m_run = -inf -> 0
        m_run[r] = m_new;
      }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float p = exp2f(s[n][e] - m_use[e >> 1]);
          s[n][e] = p;
          ls[e >> 1] += p;
          if constexpr (DUAL) {
            const float w = p * (y1[n][e] * a.sm_scale);
            y1[n][e] = w;
            ms[e >> 1] += w;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // of this thread's columns; the quad's sums are added up at the end
        l_run[r] = l_run[r] * alpha[r] + ls[r];
        if constexpr (DUAL) mu_run[r] = mu_run[r] * alpha[r] + ms[r];
      }
      if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc_o[d][e] *= alpha[e >> 1];
            if constexpr (DUAL) acc_t[d][e] *= alpha[e >> 1];
          }
        }
      }

      PairA fp;
      float kp[2];
      a_from_acc(fp, kp, s, iv, lane);
      if constexpr (DUAL) {
        PairA fw, ft;
        float kw[2], kt[2];
        a_from_acc(fw, kw, y1, iv, lane);
        if constexpr (TKV) a_from_acc(ft, kt, s, itv, lane);
        outputs_dual<D, TKV>(acc_o, acc_t, fp, kp, fw, kw, ft, kt, aV, aTV, kr, lane);
      } else {
        outputs<D, true, false>(acc_o, fp, kp, fp, kp, aV, aV, kr, lane);
      }
    }
    if (it + 1 < n_tiles) {
      if constexpr (STAGES == 1) {
        __syncthreads();  // every warp is done with the only stage
        copy_kv(it + 1);
      }
      cp_async_wait<0>();
      split_kv(it + 1);
      __syncthreads();  // the next tile is there, and every warp is done with this one
      if (STAGES == 2 && it + 2 < n_tiles) copy_kv(it + 2);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_run[r] = quad_sum(l_run[r]);
    if constexpr (DUAL) mu_run[r] = quad_sum(mu_run[r]);
  }

  // merge the key parts of a row
  if constexpr (KG > 1) {
    if (t == 0) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = r0 + g + 8 * r;
        sRow[kg * BM + i] = m_run[r];
        sRow[(KG + kg) * BM + i] = l_run[r];
        sRow[(2 * KG + kg) * BM + i] = mu_run[r];
      }
    }
    __syncthreads();
    float f[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int i = r0 + g + 8 * r;
      float m = -INFINITY, l = 0.f, mu = 0.f;
#pragma unroll
      for (int k = 0; k < KG; ++k) m = fmaxf(m, sRow[k * BM + i]);
      const float mz = m == -INFINITY ? 0.f : m;
#pragma unroll
      for (int k = 0; k < KG; ++k) {
        const float x = exp2f(sRow[k * BM + i] - mz);
        l += x * sRow[(KG + k) * BM + i];
        mu += x * sRow[(2 * KG + k) * BM + i];
      }
      f[r] = exp2f(m_run[r] - mz);
      m_run[r] = m, l_run[r] = l, mu_run[r] = mu;
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc_o[d][e] *= f[e >> 1];
        if constexpr (DUAL) acc_t[d][e] *= f[e >> 1];
      }
    }
    merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sKV), acc_o, rg, kg, lane);
    if constexpr (DUAL) merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sKV), acc_t, rg, kg, lane);
  }
  if (kg != 0) return;

  float inv_l[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool empty = !(l_run[r] > 0.f);
    inv_l[r] = empty ? 0.f : 1.f / l_run[r];
    const float mu = DUAL ? mu_run[r] * inv_l[r] : 0.f;
    const int row = r == 0 ? row_lo : row_hi;
    if (t == 0 && row < L) {
      a.lse[(size_t)bh * L + row] = empty ? INFINITY : (m_run[r] + log2f(l_run[r]));
      if constexpr (DUAL) a.mu[(size_t)bh * L + row] = mu;
    }
    if constexpr (DUAL) {  // tO = tO' / l - mu O; 1 / l follows in the store
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        acc_t[d][2 * r] -= mu * acc_o[d][2 * r];
        acc_t[d][2 * r + 1] -= mu * acc_o[d][2 * r + 1];
      }
    }
  }
  store_strip<D>(reinterpret_cast<float*>(a.o) + head_off, acc_o, inv_l, row_lo, L, lane);
  if constexpr (DUAL) store_strip<D>(reinterpret_cast<float*>(a.to) + head_off, acc_t, inv_l, row_lo, L, lane);
}

template <int D, bool DUAL, bool TKV, int RG, int KG>
int launch_one(const jvpfa_fwd_args& a, cudaStream_t stream) {
  using C = FwdCfg<D, DUAL, TKV, RG, KG>;
  static_assert(C::smem <= 227 * 1024, "shared memory of one CTA");
  auto kern = fwd_fp32_kernel<D, DUAL, TKV, RG, KG>;
  static SmemOptIn opt_in;
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), C::smem)) return JVPFA_ERR_CUDA;
  kern<<<dim3((a.L + C::BM - 1) / C::BM, a.B * a.H), C::NT, C::smem, stream>>>(a);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch fwd_fp32");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <int D>
int launch_d(const jvpfa_fwd_args& a, cudaStream_t s) {
  return dispatch_split<D>(a.B, a.H, a.L, [&](auto rg, auto kg) {
    constexpr int RG = decltype(rg)::value, KG = decltype(kg)::value;
    if (!a.tq) return launch_one<D, false, false, RG, KG>(a, s);
    return a.flags & JVPFA_ZERO_TKV ? launch_one<D, true, false, RG, KG>(a, s) : launch_one<D, true, true, RG, KG>(a, s);
  });
}

}  // namespace

int launch_fwd_fp32(const jvpfa_fwd_args& a, cudaStream_t s) {
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
