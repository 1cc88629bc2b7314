// Fused primal (+ tangent) attention forward on warp-level tensor-core MMAs.
//
// A CTA of RG x KG warps owns 16*RG query rows of one (batch, head).  Warp (rg, kg) owns 16 of the rows and the kg-th part
// of every key tile: it keeps a running maximum, denominator, mu and output of its own over its keys, and the KG partial
// results of a row are merged once, through shared memory, when the keys are through.  K, tK, V, tV tiles stream through
// a cp.async ring in shared memory.  Per tile the warp forms S = Q K^T and tS = tQ K^T + Q tK^T in registers, applies the
// mask / bias, runs the online softmax (running max m, denominator l and mu = sum P*tS) and feeds P and P*tS straight
// from the accumulator registers into the second set of MMAs (O += P V, tO' += (P*tS) V + P tV).
// Epilogue: O = acc/l, tO = tO'/l - (mu/l) O, lse = m + log2(l)  (base 2, scaled scores).
//
// Math follows upstream's _attn_fwd_inner (jvp_flash_attention/jvp_attention.py:125-336) and the
// epilogue at jvp_attention.py:1011-1033, with two deliberate differences: the additive bias
// is applied as scale*QK^T + bias (SDPA semantics; upstream scales the bias too,
// jvp_attention.py:247-251), and boolean masking uses -inf rather than adding -100.
//
// It serves fp32 and what the tcgen05 kernels do not take of the 16-bit types; with many rows, and where that is faster, the
// form with one warp for each 16 rows does instead (fwd_rows.cu; common.cuh says where the lines lie).
// What bounds it: mma.sync, at 512 (TF32) or 1024 (16-bit) multiply-adds per clock and SM, measured; an fp32 product is
// three TF32 instructions.  One instruction occupies its quarter of the SM for 8 cycles and returns after 21, and the
// fp32 products of one accumulator are a chain, so the split matters: 64 rows x D=128 fp32 fill the shared memory of an
// SM, and with one warp for each 16 rows (KG = 1) a quarter had a single warp to wait for.  With KG = 2 it has two, and
// shapes with few row tiles use shorter ones with more key parts (see launch_d) instead of leaving SMs idle.
#include <type_traits>

#include "common.cuh"

namespace jvpfa {

template <typename T, int D, int RG, int KG>
struct FwdCfg {
  static constexpr int BM = 16 * RG;
  static constexpr int NTHREADS = 32 * RG * KG;
  // keys of a warp per tile: enough for one contraction step of the second products; two where the tile fits twice
  static constexpr int BN = Elem<T>::k16 ? (D > 64 ? 32 : 64) : (KG >= 8 ? 64 : 32);
  static constexpr int BW = BN / KG;
  static constexpr int LD = D + Elem<T>::kPad;
  static constexpr int STAGES = (!Elem<T>::k16 && D > 64 && BN > 32) ? 1 : 2;
  static constexpr size_t tiles(bool dual, bool tkv) {
    const size_t ring = sizeof(T) * (size_t)STAGES * BN * LD * (tkv ? 4 : 2);
    const size_t merge = sizeof(float) * (size_t)(RG * KG / 2) * 16 * D * (dual ? 2 : 1);  // reuses the ring
    return ring > merge ? ring : merge;
  }
  static constexpr size_t smem(bool dual, bool tkv) {
    return sizeof(T) * (size_t)BM * LD * (dual ? 2 : 1) + tiles(dual, tkv) + sizeof(float) * 3 * KG * BM;
  }
};

// TKV: K and V have tangents (JVPFA_ZERO_TKV leaves them, and two of the six products, out).
// TILES: parts of key tiles without a true mask entry are left out (dead_keys).
template <typename T, int D, bool DUAL, bool TKV, int RG, int KG, bool TILES>
__global__ void __launch_bounds__(32 * RG * KG) fwd_generic_kernel(const jvpfa_fwd_args a) {
  using C = FwdCfg<T, D, RG, KG>;
  constexpr int BM = C::BM, BN = C::BN, BW = C::BW, LD = C::LD, NT = C::NTHREADS, STAGES = C::STAGES;
  constexpr int KS = Elem<T>::kKStep;
  constexpr int NS = BW / 8;   // score n-tiles per warp row-strip
  constexpr int ND = D / 8;    // output n-tiles
  constexpr int NKV = TKV ? 4 : 2;
  static_assert(BW % KS == 0, "a warp's keys are whole contraction steps");

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sQ = reinterpret_cast<T*>(smem_raw);
  T* sTQ = sQ + BM * LD;  // only valid when DUAL
  T* sKV = sQ + BM * LD * (DUAL ? 2 : 1);
  float* sRow = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(sKV) + C::tiles(DUAL, TKV));  // [3][KG][BM]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  // Heaviest causal tiles (largest m0) are scheduled first.
  const int mt = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int m0 = mt * BM;

  const size_t head_off = (size_t)bh * L * D;
  // the six inputs may share a strided (batch, head, row) layout (in_stride, elements; all zero = row-major)
  const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
  const long long in_off = strided ? (long long)b * a.in_stride[0] + (long long)h * a.in_stride[1] : (long long)head_off;
  const long long in_rs = strided ? a.in_stride[2] : D;
  const T* gQ = reinterpret_cast<const T*>(a.q) + in_off;
  const T* gK = reinterpret_cast<const T*>(a.k) + in_off;
  const T* gV = reinterpret_cast<const T*>(a.v) + in_off;
  const T* gTQ = DUAL ? reinterpret_cast<const T*>(a.tq) + in_off : nullptr;
  const T* gTK = TKV ? reinterpret_cast<const T*>(a.tk) + in_off : nullptr;
  const T* gTV = TKV ? reinterpret_cast<const T*>(a.tv) + in_off : nullptr;

  const MaskView mv = make_mask_view(a.mask, b, h, L);

  int n_end = L;
  if (mv.kind == JVPFA_MASK_CAUSAL) n_end = min(L, m0 + BM);
  if (mv.kind == JVPFA_MASK_KVLEN) n_end = min(L, mv.kv_len);
  const int n_tiles = (n_end + BN - 1) / BN;

  auto stage_kv = [&](int stage, int n0) {
    T* base = sKV + (size_t)stage * NKV * BN * LD;
    stage_tile<T, BN, D, NT>(base, gK, n0, L, tid, in_rs);
    stage_tile<T, BN, D, NT>(base + BN * LD, gV, n0, L, tid, in_rs);
    if constexpr (TKV) {
      stage_tile<T, BN, D, NT>(base + 2 * BN * LD, gTK, n0, L, tid, in_rs);
      stage_tile<T, BN, D, NT>(base + 3 * BN * LD, gTV, n0, L, tid, in_rs);
    }
  };

  // Prologue: Q (+tQ) and the first K/V tile in one cp.async group.
  stage_tile<T, BM, D, NT>(sQ, gQ, m0, L, tid, in_rs);
  if constexpr (DUAL) stage_tile<T, BM, D, NT>(sTQ, gTQ, m0, L, tid, in_rs);
  if (STAGES == 2 && n_tiles > 0) stage_kv(0, 0);
  cp_async_commit();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16;
  const int row_lo = m0 + r0 + g, row_hi = row_lo + 8;

  float acc_o[ND][4];
  float acc_t[DUAL ? ND : 1][4];
#pragma unroll
  for (int i = 0; i < ND; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc_o[i][j] = 0.f;
      if constexpr (DUAL) acc_t[i][j] = 0.f;
    }
  }
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.f, 0.f};
  float mu_run[2] = {0.f, 0.f};

  for (int it = 0; it < n_tiles; ++it) {
    int stage = 0;
    if constexpr (STAGES == 2) {
      if (it + 1 < n_tiles) stage_kv((it + 1) & 1, (it + 1) * BN);
      cp_async_commit();
      cp_async_wait<1>();
      stage = it & 1;
    } else {
      stage_kv(0, it * BN);
      cp_async_commit();
      cp_async_wait<0>();
    }
    __syncthreads();

    const int n0 = it * BN + kg * BW;  // this warp's keys of the tile
    // (a part beyond the end, or above the diagonal of the warp's rows, is nobody's work; the barrier below is everybody's)
    if (n0 < n_end && !(mv.kind == JVPFA_MASK_CAUSAL && n0 > m0 + r0 + 15) && !(TILES && dead_keys(a, b, h, m0, n0, min(n0 + BW, n_end)))) {
    const T* sK = sKV + (size_t)stage * NKV * BN * LD + kg * BW * LD;
    const T* sV = sK + BN * LD;
    const T* sTK = sK + 2 * BN * LD;
    const T* sTV = sK + 3 * BN * LD;

    // ---- user mask: fetched ahead of the products that hide its latency ----
    const bool full_tile = (mv.kind == JVPFA_MASK_NONE && n0 + BW <= L && m0 + BM <= L) ||
                           (mv.kind == JVPFA_MASK_CAUSAL && n0 + BW - 1 <= m0 + r0 && m0 + BM <= L) ||
                           (mv.kind == JVPFA_MASK_KVLEN && n0 + BW <= mv.kv_len && m0 + BM <= L);
    bool ok[NS][4];
    float bias[NS][4];
    if (!full_tile) {
#pragma unroll
      for (int nt = 0; nt < NS; ++nt) {
        mv.pair(row_lo, n0 + nt * 8 + 2 * t, &ok[nt][0], &bias[nt][0]);
        mv.pair(row_hi, n0 + nt * 8 + 2 * t, &ok[nt][2], &bias[nt][2]);
      }
    }

    // ---- scores ----
    float s[NS][4];
    float ts[DUAL ? NS : 1][4];
#pragma unroll
    for (int i = 0; i < NS; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = 0.f;
        if constexpr (DUAL) ts[i][j] = 0.f;
      }
    }
#pragma unroll 4
    for (int k0 = 0; k0 < D; k0 += KS) {
      FragA<T> fq, ftq;
      load_a<T>(fq, sQ, LD, r0, k0, lane);
      if constexpr (DUAL) load_a<T>(ftq, sTQ, LD, r0, k0, lane);
      FragB<T> fk[NS], ftk[TKV ? NS : 1];
#pragma unroll
      for (int nt = 0; nt < NS; ++nt) {
        load_b_nt<T>(fk[nt], sK, LD, nt * 8, k0, lane);
        if constexpr (TKV) load_b_nt<T>(ftk[nt], sTK, LD, nt * 8, k0, lane);
      }
      auto pass = [&](auto P) {
#pragma unroll
        for (int nt = 0; nt < NS; ++nt) {
          mma_pass<P()>(s[nt], fq, fk[nt]);
          if constexpr (DUAL) mma_pass<P()>(ts[nt], ftq, fk[nt]);
        }
        if constexpr (TKV) {
#pragma unroll
          for (int nt = 0; nt < NS; ++nt) mma_pass<P()>(ts[nt], fq, ftk[nt]);
        }
      };
      pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
    }

    // ---- mask / bias, move to the base-2 domain ----
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < NS; ++nt) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // accumulator elements 2r, 2r+1: row_lo / row_hi, keys j, j + 1
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int e = 2 * r + c;
          float x = s[nt][e] * scale_log2;
          if (!full_tile) {
            if (ok[nt][e]) {
              x += bias[nt][e] * kLog2e;
            } else {
              x = -INFINITY;
              if constexpr (DUAL) ts[nt][e] = 0.f;
            }
          }
          s[nt][e] = x;
          mx[r] = fmaxf(mx[r], x);
        }
      }
    }
    float alpha[2], m_use[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      mx[r] = quad_max(mx[r]);
      const float m_new = fmaxf(m_run[r], mx[r]);
      m_use[r] = (m_new == -INFINITY) ? 0.f : m_new;
      alpha[r] = exp2f(m_run[r] - m_use[r]);  // m_run = -inf -> 0
      m_run[r] = m_new;
    }
    float ls[2] = {0.f, 0.f}, ms[2] = {0.f, 0.f};
#pragma unroll
    for (int nt = 0; nt < NS; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p = exp2f(s[nt][e] - m_use[e >> 1]);
        s[nt][e] = p;
        ls[e >> 1] += p;
        if constexpr (DUAL) {
          const float w = p * (ts[nt][e] * a.sm_scale);
          ts[nt][e] = w;
          ms[e >> 1] += w;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      l_run[r] = l_run[r] * alpha[r] + quad_sum(ls[r]);
      if constexpr (DUAL) mu_run[r] = mu_run[r] * alpha[r] + quad_sum(ms[r]);
    }
#pragma unroll
    for (int dt = 0; dt < ND; ++dt) {
      acc_o[dt][0] *= alpha[0];
      acc_o[dt][1] *= alpha[0];
      acc_o[dt][2] *= alpha[1];
      acc_o[dt][3] *= alpha[1];
      if constexpr (DUAL) {
        acc_t[dt][0] *= alpha[0];
        acc_t[dt][1] *= alpha[0];
        acc_t[dt][2] *= alpha[1];
        acc_t[dt][3] *= alpha[1];
      }
    }

    // ---- second MMAs: contraction over the keys of this tile ----
    // fp32: the tensor core adds into its fp32 accumulator with truncation; over a thousand keys that bias reaches
    // ~1e-5.  Each contraction step is therefore formed in fresh registers and added to the running sums rounded.
#pragma unroll
    for (int kk = 0; kk < BW / KS; ++kk) {
      FragA<T> fp, fw;
      a_from_acc<T>(fp, s, kk);
      if constexpr (DUAL) a_from_acc<T>(fw, ts, kk);
      constexpr int G = 2;  // output tiles at a time
#pragma unroll
      for (int d0 = 0; d0 < ND; d0 += G) {
        FragB<T> fv[G], ftv[TKV ? G : 1];
        float xo[G][4], xt[DUAL ? G : 1][4];
#pragma unroll
        for (int i = 0; i < G; ++i) {
          load_b_nn<T>(fv[i], sV, LD, kk * KS, (d0 + i) * 8, lane);
          if constexpr (TKV) load_b_nn<T>(ftv[i], sTV, LD, kk * KS, (d0 + i) * 8, lane);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            xo[i][e] = Elem<T>::k16 ? acc_o[d0 + i][e] : 0.f;
            if constexpr (DUAL) xt[i][e] = Elem<T>::k16 ? acc_t[d0 + i][e] : 0.f;
          }
        }
        auto pass = [&](auto P) {
#pragma unroll
          for (int i = 0; i < G; ++i) {
            mma_pass<P()>(xo[i], fp, fv[i]);
            if constexpr (DUAL) mma_pass<P()>(xt[i], fw, fv[i]);
          }
          if constexpr (TKV) {
#pragma unroll
            for (int i = 0; i < G; ++i) mma_pass<P()>(xt[i], fp, ftv[i]);
          }
        };
        pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
#pragma unroll
        for (int i = 0; i < G; ++i) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            acc_o[d0 + i][e] = Elem<T>::k16 ? xo[i][e] : acc_o[d0 + i][e] + xo[i][e];
            if constexpr (DUAL) acc_t[d0 + i][e] = Elem<T>::k16 ? xt[i][e] : acc_t[d0 + i][e] + xt[i][e];
          }
        }
      }
    }
    }  // this warp's part of the tile
    __syncthreads();  // every warp is done with this stage before it is refilled
  }
  cp_async_wait<0>();
  __syncthreads();

  // ---- merge the key parts of a row ----
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
    for (int dt = 0; dt < ND; ++dt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc_o[dt][e] *= f[e >> 1];
        if constexpr (DUAL) acc_t[dt][e] *= f[e >> 1];
      }
    }
    merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sKV), acc_o, rg, kg, lane);
    if constexpr (DUAL) merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sKV), acc_t, rg, kg, lane);
  }

  // ---- epilogue ----
  float inv_l[2], mu_n[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool empty = !(l_run[r] > 0.f);
    inv_l[r] = empty ? 0.f : 1.f / l_run[r];
    mu_n[r] = DUAL ? mu_run[r] * inv_l[r] : 0.f;
    const int row = r == 0 ? row_lo : row_hi;
    if (kg == 0 && t == 0 && row < L) {
      a.lse[(size_t)bh * L + row] = empty ? INFINITY : (m_run[r] + log2f(l_run[r]));
      if constexpr (DUAL) a.mu[(size_t)bh * L + row] = mu_n[r];
    }
  }
  // Stage the output tiles through the (now idle) Q / tQ buffers for 16-byte coalesced stores.
  if (kg == 0) {
#pragma unroll
  for (int dt = 0; dt < ND; ++dt) {
    float o0 = acc_o[dt][0] * inv_l[0], o1 = acc_o[dt][1] * inv_l[0];
    float o2 = acc_o[dt][2] * inv_l[1], o3 = acc_o[dt][3] * inv_l[1];
    const int c = dt * 8 + 2 * t;
    T* plo = sQ + (r0 + g) * LD + c;
    T* phi = plo + 8 * LD;
    plo[0] = Elem<T>::from_float(o0);
    plo[1] = Elem<T>::from_float(o1);
    phi[0] = Elem<T>::from_float(o2);
    phi[1] = Elem<T>::from_float(o3);
    if constexpr (DUAL) {
      T* qlo = sTQ + (r0 + g) * LD + c;
      T* qhi = qlo + 8 * LD;
      qlo[0] = Elem<T>::from_float(acc_t[dt][0] * inv_l[0] - mu_n[0] * o0);
      qlo[1] = Elem<T>::from_float(acc_t[dt][1] * inv_l[0] - mu_n[0] * o1);
      qhi[0] = Elem<T>::from_float(acc_t[dt][2] * inv_l[1] - mu_n[1] * o2);
      qhi[1] = Elem<T>::from_float(acc_t[dt][3] * inv_l[1] - mu_n[1] * o3);
    }
  }
  }
  __syncthreads();
  {
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int VPR = D / VEC;
    T* gO = reinterpret_cast<T*>(a.o) + head_off;
    T* gTO = DUAL ? reinterpret_cast<T*>(a.to) + head_off : nullptr;
    for (int idx = tid; idx < BM * VPR; idx += NT) {
      const int r = idx / VPR, c = (idx - r * VPR) * VEC;
      const int row = m0 + r;
      if (row < L) {
        *reinterpret_cast<uint4*>(gO + (size_t)row * D + c) = *reinterpret_cast<const uint4*>(sQ + r * LD + c);
        if constexpr (DUAL)
          *reinterpret_cast<uint4*>(gTO + (size_t)row * D + c) =
              *reinterpret_cast<const uint4*>(sTQ + r * LD + c);
      }
    }
  }
}

template <typename T, int D, bool DUAL, bool TKV, int RG, int KG, bool TILES = false>
static int launch_one(const jvpfa_fwd_args& a, cudaStream_t stream) {
  if constexpr (!Elem<T>::k16 && !TILES)
    if (with_tiles(a)) return launch_one<T, D, DUAL, TKV, RG, KG, true>(a, stream);
  using C = FwdCfg<T, D, RG, KG>;
  constexpr size_t smem = C::smem(DUAL, TKV);
  static_assert(smem <= 227 * 1024, "shared memory of one CTA");
  auto kern = fwd_generic_kernel<T, D, DUAL, TKV, RG, KG, TILES>;
  static SmemOptIn opt_in;
  if (!opt_in.ensure(reinterpret_cast<const void*>(kern), smem)) return JVPFA_ERR_CUDA;
  dim3 grid((a.L + C::BM - 1) / C::BM, a.B * a.H);
  kern<<<grid, C::NTHREADS, smem, stream>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch fwd_generic");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <typename T, int D, int RG, int KG>
static int launch_split(const jvpfa_fwd_args& a, cudaStream_t s) {
  if (!a.tq) return launch_one<T, D, false, false, RG, KG>(a, s);
  if constexpr (std::is_same_v<T, float>)  // (the only type the flag is accepted for)
    if (a.flags & JVPFA_ZERO_TKV) return launch_one<T, D, true, false, RG, KG>(a, s);
  return launch_one<T, D, true, true, RG, KG>(a, s);
}

// Rows x key parts of a CTA: row_groups.
template <typename T, int D>
static int launch_d(const jvpfa_fwd_args& a, cudaStream_t s) {
  const long long rows16 = tiles16(a.B, a.H, a.L);
  if (rows16 >= kFwdRowsFrom<T, D> && !(a.flags & JVPFA_ZERO_TKV) && (!a.tq || kFwdRowsDual<T, D>)) return launch_fwd_rows(a, s);
  if constexpr (!Elem<T>::k16) {
    const int rg = row_groups(a.B, a.H, a.L, a.tq != nullptr, a.mask.kind == JVPFA_MASK_CAUSAL, kFwdRowGroups<T, D>);
    if (rg == 1) return launch_split<T, D, 1, 8>(a, s);
    if (rg == 2) return launch_split<T, D, 2, 4>(a, s);
  }
  return launch_split<T, D, 4, 2>(a, s);
}

template <typename T>
static int launch_t(const jvpfa_fwd_args& a, cudaStream_t s) {
  switch (a.D) {
    case 32:
      return launch_d<T, 32>(a, s);
    case 64:
      return launch_d<T, 64>(a, s);
    case 128:
      return launch_d<T, 128>(a, s);
    default:
      return JVPFA_ERR_SHAPE;
  }
}

int launch_fwd_generic(const jvpfa_fwd_args& a, cudaStream_t s) {
  switch (a.dtype) {
    case JVPFA_BF16:
      return launch_t<__nv_bfloat16>(a, s);
    case JVPFA_FP16:
      return launch_t<__half>(a, s);
    case JVPFA_FP32:
      return launch_t<float>(a, s);
    case JVPFA_FP32_TF32:
      return launch_t<tf32x1>(a, s);
    default:
      return JVPFA_ERR_DTYPE;
  }
}

}  // namespace jvpfa
