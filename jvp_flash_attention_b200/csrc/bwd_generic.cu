// Backward of  <gO, O> + <gtO, tO>  with respect to q, k, v on warp-level tensor-core MMAs.
//
// Per head, with s = sm_scale, S = s Q K^T + bias, P = softmax(S), tS = s (tQ K^T + Q tK^T),
// mu = rowsum(P*tS), O = P V, tO = (P*(tS - mu)) V + P tV, and cotangents gO, G = gtO:
//
//   delta = rowsum(gO*O)   eps = rowsum(G*O)   cterm = rowsum(G*tO) - eps*mu     (preprocess)
//   dP = gO V^T   E = G V^T   F = G tV^T
//   gtS = P*(E - eps)
//   gS  = P*( E*(tS - mu) - eps*tS + F + dP - delta - cterm )
//   dV = P^T gO + (P*(tS - mu))^T G
//   dQ = s (gS K + gtS tK)          dK = s (gS^T Q + gtS^T tQ)
//
// With G absent this reduces to the flash-attention-2 backward that upstream implements in
// _attn_bwd_dkdv / _attn_bwd_dq (jvp_flash_attention/jvp_attention.py:1415-1707).  Like upstream
// (jvp_attention.py:2008-2233) the work is split into a kernel that owns a key tile and loops
// over query tiles (dK, dV) and one that owns a query tile and loops over key tiles (dQ); score
// tiles are recomputed from the saved base-2 logsumexp, so results are deterministic and no
// L x L tensor or atomic accumulation is needed.
#include <type_traits>

#include "common.cuh"

namespace jvpfa {

// ----------------------------------------------------------------------------------------------
// Preprocess: three row reductions, one pass over O, tO, gO, gtO (HBM bound).
// ----------------------------------------------------------------------------------------------
template <typename T>
struct Vec16 {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};

template <typename T, int D>
__global__ void __launch_bounds__(256) pre_kernel(const jvpfa_pre_args a, long long rows) {
  behind_previous();  // (for the kernel behind this one)
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int TPR = D / VEC;  // threads per row (4..32)
  constexpr int RPB = 256 / TPR;
  const int tid = threadIdx.x;
  const long long row = (long long)blockIdx.x * RPB + tid / TPR;
  const int c = (tid % TPR) * VEC;
  const bool ok = row < rows;
  const bool has_go = a.go != nullptr, has_g = a.gto != nullptr;
  // dQ's accumulation buffer, cleared on the way: one launch and its gap less than a memset of its own
  if (ok && a.dq_accum != nullptr) {
    float4* z = reinterpret_cast<float4*>(a.dq_accum + (size_t)row * D + c);
#pragma unroll
    for (int i = 0; i < VEC / 4; ++i) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  float d = 0.f, e = 0.f, dd = 0.f;
  if (ok) {
    const size_t off = (size_t)row * D + c;
    uint4 raw = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.o) + off);
    const Vec16<T>& vo = *reinterpret_cast<const Vec16<T>*>(&raw);
    if (has_go) {
      uint4 r2 = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.go) + off);
      const Vec16<T>& vg = *reinterpret_cast<const Vec16<T>*>(&r2);
#pragma unroll
      for (int i = 0; i < VEC; ++i) d += Elem<T>::to_float(vo.v[i]) * Elem<T>::to_float(vg.v[i]);
    }
    if (has_g) {
      uint4 r3 = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.gto) + off);
      uint4 r4 = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(a.to) + off);
      const Vec16<T>& vg = *reinterpret_cast<const Vec16<T>*>(&r3);
      const Vec16<T>& vt = *reinterpret_cast<const Vec16<T>*>(&r4);
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const float gg = Elem<T>::to_float(vg.v[i]);
        e += gg * Elem<T>::to_float(vo.v[i]);
        dd += gg * Elem<T>::to_float(vt.v[i]);
      }
    }
  }
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) {
    d += __shfl_xor_sync(0xffffffffu, d, o);
    e += __shfl_xor_sync(0xffffffffu, e, o);
    dd += __shfl_xor_sync(0xffffffffu, dd, o);
  }
  if (ok && (tid % TPR) == 0) {
    a.delta[row] = d;
    a.eps[row] = e;
    a.cterm[row] = has_g ? dd - e * a.mu[row] : 0.f;
  }
}

template <typename T, int D>
static int launch_pre_one(const jvpfa_pre_args& a, cudaStream_t stream) {
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int RPB = 256 / (D / VEC);
  const long long rows = (long long)a.B * a.H * a.L;
  const long long blocks = (rows + RPB - 1) / RPB;
  pre_kernel<T, D><<<(unsigned)blocks, 256, 0, stream>>>(a, rows);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch pre_kernel");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <typename T>
static int launch_pre_t(const jvpfa_pre_args& a, cudaStream_t s) {
  switch (a.D) {
    case 32:
      return launch_pre_one<T, 32>(a, s);
    case 64:
      return launch_pre_one<T, 64>(a, s);
    case 128:
      return launch_pre_one<T, 128>(a, s);
    default:
      return JVPFA_ERR_SHAPE;
  }
}

int launch_pre(const jvpfa_pre_args& a, cudaStream_t s) {
  switch (a.dtype) {
    case JVPFA_BF16:
      return launch_pre_t<__nv_bfloat16>(a, s);
    case JVPFA_FP16:
      return launch_pre_t<__half>(a, s);
    case JVPFA_FP32:
    case JVPFA_FP32_TF32:  // no products in this kernel
      return launch_pre_t<float>(a, s);
    default:
      return JVPFA_ERR_DTYPE;
  }
}

// ----------------------------------------------------------------------------------------------
// Main kernels.  A CTA of RG x KG warps owns 16*RG rows (keys for dK / dV, queries for dQ) and loops over tiles of the
// other side; warp (rg, kg) owns 16 of the rows and the kg-th part of every loop tile, sums its own dK, dV or dQ, and the
// KG partial sums are added once at the end (a fixed order: results stay reproducible bit for bit).  As in the forward
// (fwd_generic.cu) the bound is mma.sync, three instructions for an fp32 product, and the split puts two warps on each
// quarter of an SM that shared memory would otherwise leave with one, and lets small shapes use more SMs.
//
// All score products of a tile are formed in two sweeps over D, {S, tS} and {E, F + dP}, so that an operand fragment is
// read and split once for everything it multiplies.
// ----------------------------------------------------------------------------------------------
template <typename T, int D, int RG, int KG>
struct BwdCfg {
  static constexpr int OWN = 16 * RG;  // rows owned by the CTA
  static constexpr int NTHREADS = 32 * RG * KG;
  static constexpr int LOOP = Elem<T>::k16 ? (D > 64 ? 32 : 64) : (KG >= 8 ? 64 : 32);
  static constexpr int LW = LOOP / KG;  // loop rows of a warp
  static constexpr int LD = D + Elem<T>::kPad;
  static constexpr int STAGES = (!Elem<T>::k16 && D > 64 && (RG >= 4 || LOOP > 32)) ? 1 : 2;
  static constexpr int NSTAT = 5;  // lse, delta, eps, cterm, mu
  // own_tiles / loop_tiles = number of [rows][D] operand tiles of each kind; outs = accumulators that are merged
  static constexpr size_t ring(int loop_tiles) {
    const size_t r = sizeof(T) * (size_t)STAGES * loop_tiles * LOOP * LD;
    const size_t merge = sizeof(float) * (size_t)(RG * KG / 2) * 16 * D;  // reuses the ring
    return r > merge ? r : merge;
  }
  static constexpr size_t smem(int own_tiles, int loop_tiles, bool stats) {
    return sizeof(T) * (size_t)own_tiles * OWN * LD + ring(loop_tiles) + (stats ? sizeof(float) * STAGES * NSTAT * LOOP : 0);
  }
};

// x += A0 B0^T and, where asked for, y += A1 B0^T (HAS_Y1) + A0 B1^T (HAS_Y2); rows r0.. of A0 / A1, all operands D-contiguous.
// {S, tS} with (Q, tQ; K, tK), {E, F + dP} with (V, tV; G, gO) of the side in question.
// TF32: the two products of y have an accumulator each and are added once, rounded (see gemm_out): in a single one the larger
// of the two was truncated by the adds of both (tangents of a tenth, D128 L500 causal: dQ 2.0e-6 -> 2.7e-6).
template <typename T, int D, int NT_, bool HAS_Y1, bool HAS_Y2>
__device__ __forceinline__ void gemm_pair(float (*x)[4], float (*y)[4], const T* sA0, const T* sA1, const T* sB0, const T* sB1, int ld,
                                          int r0, int lane) {
  constexpr int KS = Elem<T>::kKStep;
  constexpr bool kApart = HAS_Y1 && HAS_Y2 && !Elem<T>::k16;
  float apart[kApart ? NT_ : 1][4];
  if constexpr (kApart) zero_acc<NT_>(apart);
#pragma unroll 4
  for (int k0 = 0; k0 < D; k0 += KS) {
    FragA<T> a0, a1;
    load_a<T>(a0, sA0, ld, r0, k0, lane);
    if constexpr (HAS_Y1) load_a<T>(a1, sA1, ld, r0, k0, lane);
    FragB<T> b0[NT_], b1[HAS_Y2 ? NT_ : 1];
#pragma unroll
    for (int nt = 0; nt < NT_; ++nt) {
      load_b_nt<T>(b0[nt], sB0, ld, nt * 8, k0, lane);
      if constexpr (HAS_Y2) load_b_nt<T>(b1[nt], sB1, ld, nt * 8, k0, lane);
    }
    auto pass = [&](auto P) {
#pragma unroll
      for (int nt = 0; nt < NT_; ++nt) {
        mma_pass<P()>(x[nt], a0, b0[nt]);
        if constexpr (HAS_Y1) mma_pass<P()>(y[nt], a1, b0[nt]);
      }
      if constexpr (HAS_Y2) {
#pragma unroll
        for (int nt = 0; nt < NT_; ++nt) mma_pass<P()>(kApart ? apart[nt] : y[nt], a0, b1[nt]);
      }
    };
    pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
  }
  if constexpr (kApart) {
#pragma unroll
    for (int nt = 0; nt < NT_; ++nt) {
#pragma unroll
      for (int e = 0; e < 4; ++e) y[nt][e] += apart[nt][e];
    }
  }
}

// out[D/8][4] += A0 B0 (+ A1 B1): A from accumulator tiles (16 x KROWS), B = [k][d] tiles, d contiguous.
// fp32: the tensor core adds into its fp32 accumulator with truncation, and hundreds of such adds into one long-lived
// accumulator show up as a bias of ~1e-5.  Each contraction step is therefore formed in fresh registers and added rounded.
template <typename T, int D, int KROWS, bool HAS_0, bool HAS_1>
__device__ __forceinline__ void gemm_out(float (*out)[4], const float (*at0)[4], const float (*at1)[4], const T* sB0, const T* sB1,
                                         int ld, int lane) {
  constexpr int KS = Elem<T>::kKStep;
  constexpr int G = 4;  // output tiles at a time
#pragma unroll
  for (int kk = 0; kk < KROWS / KS; ++kk) {
    FragA<T> a0, a1;
    if constexpr (HAS_0) a_from_acc<T>(a0, at0, kk);
    if constexpr (HAS_1) a_from_acc<T>(a1, at1, kk);
#pragma unroll
    for (int d0 = 0; d0 < D / 8; d0 += G) {
      FragB<T> b0[G], b1[G];
      float tmp[G][4];
#pragma unroll
      for (int i = 0; i < G; ++i) {
        if constexpr (HAS_0) load_b_nn<T>(b0[i], sB0, ld, kk * KS, (d0 + i) * 8, lane);
        if constexpr (HAS_1) load_b_nn<T>(b1[i], sB1, ld, kk * KS, (d0 + i) * 8, lane);
#pragma unroll
        for (int e = 0; e < 4; ++e) tmp[i][e] = Elem<T>::k16 ? out[d0 + i][e] : 0.f;
      }
      auto pass = [&](auto P) {
        if constexpr (HAS_0) {
#pragma unroll
          for (int i = 0; i < G; ++i) mma_pass<P()>(tmp[i], a0, b0[i]);
        }
        if constexpr (HAS_1) {
#pragma unroll
          for (int i = 0; i < G; ++i) mma_pass<P()>(tmp[i], a1, b1[i]);
        }
      };
      pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
#pragma unroll
      for (int i = 0; i < G; ++i) {
#pragma unroll
        for (int e = 0; e < 4; ++e) out[d0 + i][e] = Elem<T>::k16 ? tmp[i][e] : out[d0 + i][e] + tmp[i][e];
      }
    }
  }
}

// ---- dK, dV: CTA owns 64 keys, loops over query tiles.  Tiles are held transposed
// (rows = keys, columns = queries) so that P^T etc. feed the second MMAs from registers. ----
// fp32 (and TF32) at head dimension 32 with tangents: 128 registers, for two CTAs of 64 rows on an SM; the compiler would take
// up to 163 (B2 H8 L2048, dQ through tO 1025 -> 839 us with what then spills).
template <typename T, int D, bool HAS_GT, int RG>
constexpr bool kTwoOnAnSm = !Elem<T>::k16 && D == 32 && HAS_GT && RG == 4;

// TKV: K and V have tangents (JVPFA_ZERO_TKV leaves out what they would be multiplied by; it comes without gO).  TILES: parts of loop tiles
// without a true mask entry are left out (dead_queries, dead_keys).
template <typename T, int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG, bool TILES>
__global__ void __launch_bounds__(32 * RG * KG, kTwoOnAnSm<T, D, HAS_GT, RG> ? 2 : 0) bwd_dkdv_kernel(const jvpfa_bwd_args a) {
  using C = BwdCfg<T, D, RG, KG>;
  constexpr int BN = C::OWN, BM = C::LOOP, LD = C::LD, NT = C::NTHREADS, STAGES = C::STAGES, LW = C::LW;
  constexpr int NQ = LW / 8;
  constexpr int ND = D / 8;
  constexpr int OWN_TILES = TKV ? 4 : 2;
  constexpr int LOOP_TILES = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0);
  static_assert(LW % Elem<T>::kKStep == 0, "a warp's loop rows are whole contraction steps");

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sK = reinterpret_cast<T*>(smem_raw);
  T* sV = sK + BN * LD;
  T* sTK = sK + 2 * BN * LD;  // TKV only
  T* sTV = sK + 3 * BN * LD;  // TKV only
  T* sLoop = sK + OWN_TILES * BN * LD;
  float* sStat = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(sLoop) + C::ring(LOOP_TILES));

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  const int n0 = blockIdx.x * BN;
  const size_t head_off = (size_t)bh * L * D;
  const size_t stat_off = (size_t)bh * L;

  // the six inputs may share a strided (batch, head, row) layout (in_stride, elements; all zero = row-major)
  const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
  const long long in_off = strided ? (long long)b * a.in_stride[0] + (long long)h * a.in_stride[1] : (long long)head_off;
  const long long in_rs = strided ? a.in_stride[2] : D;
  const T* gQ = reinterpret_cast<const T*>(a.q) + in_off;
  const T* gK = reinterpret_cast<const T*>(a.k) + in_off;
  const T* gV = reinterpret_cast<const T*>(a.v) + in_off;
  const T* gTQ = HAS_GT ? reinterpret_cast<const T*>(a.tq) + in_off : nullptr;
  const T* gTK = TKV ? reinterpret_cast<const T*>(a.tk) + in_off : nullptr;
  const T* gTV = TKV ? reinterpret_cast<const T*>(a.tv) + in_off : nullptr;
  const T* gGO = HAS_GO ? reinterpret_cast<const T*>(a.go) + head_off : nullptr;
  const T* gG = HAS_GT ? reinterpret_cast<const T*>(a.gto) + head_off : nullptr;

  const MaskView mv = make_mask_view(a.mask, b, h, L);

  // Query tiles that can see this key tile.
  int m_begin = 0;
  if (mv.kind == JVPFA_MASK_CAUSAL) m_begin = (n0 / BM) * BM;
  int n_tiles = (L - m_begin + BM - 1) / BM;
  if (mv.kind == JVPFA_MASK_KVLEN && n0 >= mv.kv_len) n_tiles = 0;

  auto stage_loop = [&](int stage, int m0) {
    T* base = sLoop + (size_t)stage * LOOP_TILES * BM * LD;
    int k = 0;
    stage_tile<T, BM, D, NT>(base + (k++) * BM * LD, gQ, m0, L, tid, in_rs);
    if constexpr (HAS_GO) stage_tile<T, BM, D, NT>(base + (k++) * BM * LD, gGO, m0, L, tid);
    if constexpr (HAS_GT) {
      stage_tile<T, BM, D, NT>(base + (k++) * BM * LD, gTQ, m0, L, tid, in_rs);
      stage_tile<T, BM, D, NT>(base + (k++) * BM * LD, gG, m0, L, tid);
    }
    if (tid < BM) {
      float* st = sStat + stage * C::NSTAT * BM;
      const int i = m0 + tid;
      const bool ok = i < L;
      st[0 * BM + tid] = ok ? a.lse[stat_off + i] : INFINITY;
      st[1 * BM + tid] = ok ? a.delta[stat_off + i] : 0.f;
      if constexpr (HAS_GT) {
        st[2 * BM + tid] = ok ? a.eps[stat_off + i] : 0.f;
        st[3 * BM + tid] = ok ? a.cterm[stat_off + i] : 0.f;
        st[4 * BM + tid] = ok ? a.mu[stat_off + i] : 0.f;
      }
    }
  };

  stage_tile<T, BN, D, NT>(sK, gK, n0, L, tid, in_rs);
  stage_tile<T, BN, D, NT>(sV, gV, n0, L, tid, in_rs);
  if constexpr (TKV) {
    stage_tile<T, BN, D, NT>(sTK, gTK, n0, L, tid, in_rs);
    stage_tile<T, BN, D, NT>(sTV, gTV, n0, L, tid, in_rs);
  }
  if (STAGES == 2 && n_tiles > 0) stage_loop(0, m_begin);
  cp_async_commit();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16;
  const int key_lo = n0 + r0 + g, key_hi = key_lo + 8;

  float dk[ND][4], dv[ND][4];
  zero_acc<ND>(dk);
  zero_acc<ND>(dv);

  for (int it = 0; it < n_tiles; ++it) {
    const int m0 = m_begin + it * BM;
    int stage;
    if (STAGES == 2) {
      if (it + 1 < n_tiles) stage_loop((it + 1) & 1, m0 + BM);
      cp_async_commit();
      cp_async_wait<1>();
      stage = it & 1;
    } else {
      stage_loop(0, m0);
      cp_async_commit();
      cp_async_wait<0>();
      stage = 0;
    }
    __syncthreads();

    // this warp's queries of the tile (none of them may see its keys: nothing to do)
    const int mw = m0 + kg * LW;
    if (mw < L && !(mv.kind == JVPFA_MASK_CAUSAL && mw + LW <= n0 + r0) && !(TILES && dead_queries(a, b, h, n0, mw, min(mw + LW, L)))) {
      const T* sQ = sLoop + (size_t)stage * LOOP_TILES * BM * LD + kg * LW * LD;
      const T* sGO = sQ + BM * LD;                           // HAS_GO
      const T* sTQ = sQ + (1 + (HAS_GO ? 1 : 0)) * BM * LD;  // HAS_GT
      const T* sG = sTQ + BM * LD;                           // HAS_GT
      const float* st = sStat + stage * C::NSTAT * BM + kg * LW;

      bool ok[NQ][4];  // fetched ahead of the products that hide its latency
      float bias[NQ][4];
#pragma unroll
      for (int nt = 0; nt < NQ; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = mw + nt * 8 + 2 * t + (e & 1), j = (e < 2) ? key_lo : key_hi;
          ok[nt][e] = mv.allowed(i, j);
          bias[nt][e] = ok[nt][e] ? mv.bias(i, j) : 0.f;
        }
      }
      // S^T, tS^T; E^T (or dP^T), F^T + dP^T
      float p[NQ][4], ts[NQ][4], e_[NQ][4], f[NQ][4];
      zero_acc<NQ>(p);
      zero_acc<NQ>(ts);
      zero_acc<NQ>(e_);
      zero_acc<NQ>(f);
      gemm_pair<T, D, NQ, TKV, HAS_GT>(p, ts, sK, sTK, sQ, sTQ, LD, r0, lane);
      if constexpr (HAS_GT)
        gemm_pair<T, D, NQ, TKV, HAS_GO>(e_, f, sV, sTV, sG, sGO, LD, r0, lane);
      else
        gemm_pair<T, D, NQ, false, false>(f, f, sV, sV, sGO, sGO, LD, r0, lane);

#pragma unroll
      for (int nt = 0; nt < NQ; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ci = nt * 8 + 2 * t + (e & 1);
          float pv = 0.f;
          if (ok[nt][e]) pv = exp2f(p[nt][e] * scale_log2 + bias[nt][e] * kLog2e - st[ci]);
          float sub = st[1 * BM + ci];
          if constexpr (HAS_GT) {
            const float tsv = ts[nt][e] * a.sm_scale, ev = e_[nt][e], eps = st[2 * BM + ci], mu = st[4 * BM + ci];
            sub += st[3 * BM + ci];
            f[nt][e] += ev * (tsv - mu) - eps * tsv;
            e_[nt][e] = pv * (ev - eps);  // gtS
            ts[nt][e] = pv * (tsv - mu);  // A
          }
          f[nt][e] = pv * (f[nt][e] - sub);  // gS
          p[nt][e] = pv;
        }
      }
      // dV += P^T gO + (P*(tS-mu))^T G ;  dK += gS^T Q + gtS^T tQ
      gemm_out<T, D, LW, HAS_GO, HAS_GT>(dv, p, ts, sGO, sG, LD, lane);
      gemm_out<T, D, LW, true, HAS_GT>(dk, f, e_, sQ, sTQ, LD, lane);
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  __syncthreads();
  if constexpr (KG > 1) {
    merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dk, rg, kg, lane);
    merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dv, rg, kg, lane);
  }

  // Own K / V buffers are idle now: reuse them to coalesce the stores.
  if (kg == 0) {
    acc_to_smem<T, D>(sK, LD, r0, lane, dk, a.sm_scale);
    acc_to_smem<T, D>(sV, LD, r0, lane, dv, 1.f);
  }
  __syncthreads();
  smem_tile_to_global<T, BN, D, NT>(reinterpret_cast<T*>(a.dk) + head_off, sK, LD, n0, L, tid);
  smem_tile_to_global<T, BN, D, NT>(reinterpret_cast<T*>(a.dv) + head_off, sV, LD, n0, L, tid);
}

// ---- dQ: CTA owns 64 queries, loops over key tiles (rows = queries, columns = keys). ----
template <typename T, int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG, bool TILES>
__global__ void __launch_bounds__(32 * RG * KG, kTwoOnAnSm<T, D, HAS_GT, RG> ? 2 : 0) bwd_dq_kernel(const jvpfa_bwd_args a) {
  using C = BwdCfg<T, D, RG, KG>;
  constexpr int BM = C::OWN, BN = C::LOOP, LD = C::LD, NT = C::NTHREADS, STAGES = C::STAGES, LW = C::LW;
  constexpr int NK = LW / 8;
  constexpr int ND = D / 8;
  constexpr int OWN_TILES = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0);
  constexpr int LOOP_TILES = TKV ? 4 : 2;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sQ = reinterpret_cast<T*>(smem_raw);
  T* sGO = sQ + BM * LD;                              // HAS_GO
  T* sTQ = sQ + (1 + (HAS_GO ? 1 : 0)) * BM * LD;     // HAS_GT
  T* sG = sTQ + BM * LD;                              // HAS_GT
  T* sLoop = sQ + OWN_TILES * BM * LD;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = warp % RG, kg = warp / RG;
  const int g = lane >> 2, t = lane & 3;
  const int L = a.L;
  const int bh = blockIdx.y;
  const int b = bh / a.H, h = bh - b * a.H;
  const int mt = (int)gridDim.x - 1 - (int)blockIdx.x;
  const int m0 = mt * BM;
  const size_t head_off = (size_t)bh * L * D;
  const size_t stat_off = (size_t)bh * L;

  // the six inputs may share a strided (batch, head, row) layout (in_stride, elements; all zero = row-major)
  const bool strided = (a.in_stride[0] | a.in_stride[1] | a.in_stride[2]) != 0;
  const long long in_off = strided ? (long long)b * a.in_stride[0] + (long long)h * a.in_stride[1] : (long long)head_off;
  const long long in_rs = strided ? a.in_stride[2] : D;
  const T* gQ = reinterpret_cast<const T*>(a.q) + in_off;
  const T* gK = reinterpret_cast<const T*>(a.k) + in_off;
  const T* gV = reinterpret_cast<const T*>(a.v) + in_off;
  const T* gTQ = HAS_GT ? reinterpret_cast<const T*>(a.tq) + in_off : nullptr;
  const T* gTK = TKV ? reinterpret_cast<const T*>(a.tk) + in_off : nullptr;
  const T* gTV = TKV ? reinterpret_cast<const T*>(a.tv) + in_off : nullptr;
  const T* gGO = HAS_GO ? reinterpret_cast<const T*>(a.go) + head_off : nullptr;
  const T* gG = HAS_GT ? reinterpret_cast<const T*>(a.gto) + head_off : nullptr;

  const MaskView mv = make_mask_view(a.mask, b, h, L);

  int n_end = L;
  if (mv.kind == JVPFA_MASK_CAUSAL) n_end = min(L, m0 + BM);
  if (mv.kind == JVPFA_MASK_KVLEN) n_end = min(L, mv.kv_len);
  const int n_tiles = (n_end + BN - 1) / BN;

  auto stage_loop = [&](int stage, int n0) {
    T* base = sLoop + (size_t)stage * LOOP_TILES * BN * LD;
    stage_tile<T, BN, D, NT>(base, gK, n0, L, tid, in_rs);
    stage_tile<T, BN, D, NT>(base + BN * LD, gV, n0, L, tid, in_rs);
    if constexpr (TKV) {
      stage_tile<T, BN, D, NT>(base + 2 * BN * LD, gTK, n0, L, tid, in_rs);
      stage_tile<T, BN, D, NT>(base + 3 * BN * LD, gTV, n0, L, tid, in_rs);
    }
  };

  stage_tile<T, BM, D, NT>(sQ, gQ, m0, L, tid, in_rs);
  if constexpr (HAS_GO) stage_tile<T, BM, D, NT>(sGO, gGO, m0, L, tid);
  if constexpr (HAS_GT) {
    stage_tile<T, BM, D, NT>(sTQ, gTQ, m0, L, tid, in_rs);
    stage_tile<T, BM, D, NT>(sG, gG, m0, L, tid);
  }
  if (STAGES == 2 && n_tiles > 0) stage_loop(0, 0);
  cp_async_commit();

  const float scale_log2 = a.sm_scale * kLog2e;
  const int r0 = rg * 16;
  const int row[2] = {m0 + r0 + g, m0 + r0 + g + 8};
  float lse[2], sub[2], eps[2] = {0.f, 0.f}, mu[2] = {0.f, 0.f};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const bool ok = row[r] < L;
    lse[r] = ok ? a.lse[stat_off + row[r]] : INFINITY;
    sub[r] = ok ? a.delta[stat_off + row[r]] : 0.f;
    if constexpr (HAS_GT) {
      sub[r] += ok ? a.cterm[stat_off + row[r]] : 0.f;
      eps[r] = ok ? a.eps[stat_off + row[r]] : 0.f;
      mu[r] = ok ? a.mu[stat_off + row[r]] : 0.f;
    }
  }

  float dq[ND][4];
  zero_acc<ND>(dq);

  for (int it = 0; it < n_tiles; ++it) {
    const int n0 = it * BN;
    int stage;
    if (STAGES == 2) {
      if (it + 1 < n_tiles) stage_loop((it + 1) & 1, n0 + BN);
      cp_async_commit();
      cp_async_wait<1>();
      stage = it & 1;
    } else {
      stage_loop(0, n0);
      cp_async_commit();
      cp_async_wait<0>();
      stage = 0;
    }
    __syncthreads();

    const int nw = n0 + kg * LW;  // this warp's keys of the tile
    if (nw < n_end && !(mv.kind == JVPFA_MASK_CAUSAL && nw > m0 + r0 + 15) && !(TILES && dead_keys(a, b, h, m0, nw, min(nw + LW, n_end)))) {
      const T* sK = sLoop + (size_t)stage * LOOP_TILES * BN * LD + kg * LW * LD;
      const T* sV = sK + BN * LD;
      const T* sTK = sK + 2 * BN * LD;
      const T* sTV = sK + 3 * BN * LD;

      bool ok[NK][4];  // fetched ahead of the products that hide its latency
      float bias[NK][4];
#pragma unroll
      for (int nt = 0; nt < NK; ++nt) {
        mv.pair(row[0], nw + nt * 8 + 2 * t, &ok[nt][0], &bias[nt][0]);
        mv.pair(row[1], nw + nt * 8 + 2 * t, &ok[nt][2], &bias[nt][2]);
      }
      float p[NK][4], ts[NK][4], e_[NK][4], f[NK][4];
      zero_acc<NK>(p);
      zero_acc<NK>(ts);
      zero_acc<NK>(e_);
      zero_acc<NK>(f);
      gemm_pair<T, D, NK, HAS_GT, TKV>(p, ts, sQ, sTQ, sK, sTK, LD, r0, lane);
      if constexpr (HAS_GT) {
        // E = G V^T, F = G tV^T; dP = gO V^T shares V
        gemm_pair<T, D, NK, HAS_GO, TKV>(e_, f, sG, sGO, sV, sTV, LD, r0, lane);
      } else {
        gemm_pair<T, D, NK, false, false>(f, f, sGO, sGO, sV, sV, LD, r0, lane);
      }

#pragma unroll
      for (int nt = 0; nt < NK; ++nt) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {  // accumulator elements 2r, 2r+1: one query row, keys j and j + 1
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int e = 2 * r + c;
            float pv = 0.f;
            if (ok[nt][e]) pv = exp2f(p[nt][e] * scale_log2 + bias[nt][e] * kLog2e - lse[r]);
            if constexpr (HAS_GT) {
              const float tsv = ts[nt][e] * a.sm_scale, ev = e_[nt][e];
              f[nt][e] += ev * (tsv - mu[r]) - eps[r] * tsv;
              e_[nt][e] = pv * (ev - eps[r]);  // gtS
            }
            f[nt][e] = pv * (f[nt][e] - sub[r]);  // gS
          }
        }
      }
      gemm_out<T, D, LW, true, TKV>(dq, f, e_, sK, sTK, LD, lane);  // gS K + gtS tK
    }
    __syncthreads();
  }
  cp_async_wait<0>();
  __syncthreads();
  if constexpr (KG > 1) merge_parts<RG, KG, ND>(reinterpret_cast<float4*>(sLoop), dq, rg, kg, lane);

  if (kg == 0) acc_to_smem<T, D>(sQ, LD, r0, lane, dq, a.sm_scale);
  __syncthreads();
  smem_tile_to_global<T, BM, D, NT>(reinterpret_cast<T*>(a.dq) + head_off, sQ, LD, m0, L, tid);
}

template <typename T, int D, bool HAS_GO, bool HAS_GT, bool TKV, int RG, int KG, bool TILES = false>
static int launch_bwd_one(const jvpfa_bwd_args& a, cudaStream_t stream) {
  if constexpr (!Elem<T>::k16 && !TILES)
    if (with_tiles(a)) return launch_bwd_one<T, D, HAS_GO, HAS_GT, TKV, RG, KG, true>(a, stream);
  using C = BwdCfg<T, D, RG, KG>;
  constexpr int keys = TKV ? 4 : 2, queries = 1 + (HAS_GO ? 1 : 0) + (HAS_GT ? 2 : 0);  // tiles of each side
  constexpr size_t smem_kv = C::smem(keys, queries, true);
  constexpr size_t smem_q = C::smem(queries, keys, false);
  static_assert(smem_kv <= 227 * 1024 && smem_q <= 227 * 1024, "shared memory of one CTA");
  auto k1 = bwd_dkdv_kernel<T, D, HAS_GO, HAS_GT, TKV, RG, KG, TILES>;
  auto k2 = bwd_dq_kernel<T, D, HAS_GO, HAS_GT, TKV, RG, KG, TILES>;
  static SmemOptIn opt_in1, opt_in2;
  if (!opt_in1.ensure(reinterpret_cast<const void*>(k1), smem_kv) || !opt_in2.ensure(reinterpret_cast<const void*>(k2), smem_q))
    return JVPFA_ERR_CUDA;
  dim3 grid((a.L + C::OWN - 1) / C::OWN, a.B * a.H);
  if (!(a.flags & JVPFA_SKIP_DKDV)) k1<<<grid, C::NTHREADS, smem_kv, stream>>>(a);
  if (!(a.flags & JVPFA_SKIP_DQ)) k2<<<grid, C::NTHREADS, smem_q, stream>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch bwd_generic");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

template <typename T, int D, int RG, int KG>
static int launch_bwd_split(const jvpfa_bwd_args& a, cudaStream_t s) {
  const bool go = a.go != nullptr, gt = a.gto != nullptr;
  if (go && gt) return launch_bwd_one<T, D, true, true, true, RG, KG>(a, s);
  if constexpr (std::is_same_v<T, float>)  // (the only type the flag is accepted for, and without gO)
    if (a.flags & JVPFA_ZERO_TKV) return launch_bwd_one<T, D, false, true, false, RG, KG>(a, s);
  if (gt) return launch_bwd_one<T, D, false, true, true, RG, KG>(a, s);
  return launch_bwd_one<T, D, true, false, false, RG, KG>(a, s);
}

// Rows x loop parts of a CTA, by the same rule as in the forward.
template <typename T, int D>
static int launch_bwd_d(const jvpfa_bwd_args& a, cudaStream_t s) {
  const long long rows16 = tiles16(a.B, a.H, a.L);
  if (rows16 >= kBwdRowsFrom<T, D> && (!a.gto || kBwdRowsDual<T, D>)) return launch_bwd_rows(a, s);  // (JVPFA_ZERO_TKV: fp32 with gto)
  if constexpr (!Elem<T>::k16) {
    const int rg = row_groups(a.B, a.H, a.L, a.gto != nullptr, a.mask.kind == JVPFA_MASK_CAUSAL, kBwdRowGroups<T, D>);
    if (rg == 1) return launch_bwd_split<T, D, 1, 8>(a, s);
    if (rg == 2) return launch_bwd_split<T, D, 2, 4>(a, s);
  }
  return launch_bwd_split<T, D, 4, 2>(a, s);
}

template <typename T>
static int launch_bwd_t(const jvpfa_bwd_args& a, cudaStream_t s) {
  switch (a.D) {
    case 32:
      return launch_bwd_d<T, 32>(a, s);
    case 64:
      return launch_bwd_d<T, 64>(a, s);
    case 128:
      return launch_bwd_d<T, 128>(a, s);
    default:
      return JVPFA_ERR_SHAPE;
  }
}

int launch_bwd_generic(const jvpfa_bwd_args& a, cudaStream_t s) {
  switch (a.dtype) {
    case JVPFA_BF16:
      return launch_bwd_t<__nv_bfloat16>(a, s);
    case JVPFA_FP16:
      return launch_bwd_t<__half>(a, s);
    case JVPFA_FP32:
      return launch_bwd_t<float>(a, s);
    case JVPFA_FP32_TF32:
      return launch_bwd_t<tf32x1>(a, s);
    default:
      return JVPFA_ERR_DTYPE;
  }
}

}  // namespace jvpfa
