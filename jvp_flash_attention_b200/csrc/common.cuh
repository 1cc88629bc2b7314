// Shared device helpers for the register-tiled (mma.sync) attention kernels:
// warp-level MMA fragments for bf16 / fp16 (m16n8k16) and fp32 (m16n8k8 TF32 issued
// three times on a hi/lo split, "3xTF32"), cp.async tile staging, and the mask /
// bias accessor used inside every tile loop.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/jvpfa.h"

namespace jvpfa {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// ----------------------------------------------------------------------------------------------
// Element traits
// ----------------------------------------------------------------------------------------------
template <typename T>
struct Elem;

template <>
struct Elem<__nv_bfloat16> {
  static constexpr bool k16 = true;
  static constexpr bool kSplit = false;
  static constexpr int kPad = 8;  // smem row padding in elements (keeps 16-byte rows, spreads banks)
  static constexpr int kKStep = 16;
  __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }
  __device__ static __forceinline__ __nv_bfloat16 from_float(float x) { return __float2bfloat16_rn(x); }
};

template <>
struct Elem<__half> {
  static constexpr bool k16 = true;
  static constexpr bool kSplit = false;
  static constexpr int kPad = 8;
  static constexpr int kKStep = 16;
  __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __device__ static __forceinline__ float to_float(__half x) { return __half2float(x); }
  __device__ static __forceinline__ __half from_float(float x) { return __float2half_rn(x); }
};

template <>
struct Elem<float> {
  static constexpr bool k16 = false;
  static constexpr bool kSplit = true;  // every product is three TF32 MMAs on a hi/lo split
  static constexpr int kPad = 4;
  static constexpr int kKStep = 8;
  __device__ static __forceinline__ float to_float(float x) { return x; }
  __device__ static __forceinline__ float from_float(float x) { return x; }
};

// fp32 in memory, products as one TF32 MMA (JVPFA_FP32_TF32): the precision of upstream's fp32 path, whose
// tl.dot calls run on TF32 tensor cores (jvp_attention.py:233-236, 314-322).  Relative error about 5e-4.
struct tf32x1 {
  float v;
};
template <>
struct Elem<tf32x1> {
  static constexpr bool k16 = false;
  static constexpr bool kSplit = false;
  static constexpr int kPad = 4;
  static constexpr int kKStep = 8;
  __device__ static __forceinline__ float to_float(tf32x1 x) { return x.v; }
  __device__ static __forceinline__ tf32x1 from_float(float x) { return tf32x1{x}; }
};

// ----------------------------------------------------------------------------------------------
// Raw MMA instructions.  Lane decomposition used everywhere: g = lane >> 2 (0..7), t = lane & 3.
//   C (16x8 fp32): c0=(g,2t) c1=(g,2t+1) c2=(g+8,2t) c3=(g+8,2t+1)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_16816(const __nv_bfloat16*, float c[4], const uint32_t a[4],
                                          const uint32_t b[2]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_16816(const __half*, float c[4], const uint32_t a[4],
                                          const uint32_t b[2]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_1688_tf32(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int I>
struct IntC {  // a compile-time int as an argument
  static constexpr int value = I;
  __host__ __device__ constexpr int operator()() const { return I; }
};

// Split an fp32 value into a TF32 "hi" part (11 significant bits) and the TF32 rounding of the remainder.  Dekker's
// splitting (T. J. Dekker, "A floating-point technique for extending the available precision", Numer. Math. 18, 1971)
// rounds hi on the FMA pipe, here at 2^-14 of x's magnitude: his factor of 2^13 + 1 would overflow from 2^115 on, where an
// entry must stay itself.  A tensor core ignores the low 13 bits of a TF32 operand, so half a unit of the last used bit,
// added as an integer, rounds lo.  A NaN stays one in hi.  Two cvt.rna.tf32 instead cost more issue slots than all the
// rest of a fragment (D = 128, B2 H8 L1024 with bias, primal + tangent forward: 900 us with them and the bias fetched
// behind the products, 683 us without either).
//
// Every entry has an exponent of its own, hence 22 significant bits whatever else its row or column holds, and an Inf or a
// NaN reaches only the results that it belongs to.  Pairs of fp16 numbers with one exponent for a row multiply at twice the
// rate, but leave an entry 40 bits below its row's largest nothing: one V entry of 1e8 cost the other columns of those keys
// 4e-5, one of 1e15 or Inf the keys themselves.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  constexpr float kDown = 0x1p-14f;
  const float c = __fmul_rn(x, 8193.f * kDown);  // 2^13 + 1
  const float h = __fmul_rn(__fsub_rn(c, __fmaf_rn(x, -kDown, c)), 1.f / kDown);
  hi = __float_as_uint(h);
  lo = __float_as_uint(__fsub_rn(x, h)) + 0x1000u;
}
// The same for element type T: types that multiply in one pass have no lo part.
template <typename T>
__device__ __forceinline__ void split_t(float x, uint32_t& hi, uint32_t& lo) {
  if constexpr (Elem<T>::kSplit) {
    split_tf32(x, hi, lo);
  } else {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    lo = 0u;
  }
}

// ----------------------------------------------------------------------------------------------
// Fragments.  For 16-bit types a fragment is the packed register set of m16n8k16; for fp32 it
// carries the hi and lo TF32 halves so that one logical MMA is lo*hi + hi*lo + hi*hi.
// ----------------------------------------------------------------------------------------------
template <typename T, bool k16 = Elem<T>::k16>
struct FragA;
template <typename T, bool k16 = Elem<T>::k16>
struct FragB;

template <typename T>
struct FragA<T, true> {
  uint32_t r[4];
};
template <typename T>
struct FragB<T, true> {
  uint32_t r[2];
};
template <typename T>
struct FragA<T, false> {
  uint32_t hi[4], lo[4];
};
template <typename T>
struct FragB<T, false> {
  uint32_t hi[2], lo[2];
};

template <typename T>
__device__ __forceinline__ void mma(float c[4], const FragA<T, true>& a, const FragB<T, true>& b) {
  mma_16816(static_cast<const T*>(nullptr), c, a.r, b.r);
}
template <typename T>
__device__ __forceinline__ void mma(float c[4], const FragA<T, false>& a, const FragB<T, false>& b) {
  if constexpr (Elem<T>::kSplit) {
    mma_1688_tf32(c, a.lo, b.hi);
    mma_1688_tf32(c, a.hi, b.lo);
  }
  mma_1688_tf32(c, a.hi, b.hi);
}

// One of the up to three instructions of a logical MMA: 0 = lo*hi, 1 = hi*lo, 2 = hi*hi (types that multiply in one pass
// have the last only).  Accumulators that take several products interleave the passes of all of them: an instruction
// returns after 21 cycles, and the next one on the same accumulator should be three issue slots (of 8 cycles) away.
template <int PASS, typename T>
__device__ __forceinline__ void mma_pass(float c[4], const FragA<T, true>& a, const FragB<T, true>& b) {
  if constexpr (PASS == 2) mma_16816(static_cast<const T*>(nullptr), c, a.r, b.r);
}
template <int PASS, typename T>
__device__ __forceinline__ void mma_pass(float c[4], const FragA<T, false>& a, const FragB<T, false>& b) {
  if constexpr (PASS == 2)
    mma_1688_tf32(c, a.hi, b.hi);
  else if constexpr (Elem<T>::kSplit)
    mma_1688_tf32(c, PASS == 0 ? a.lo : a.hi, PASS == 0 ? b.hi : b.lo);
}

// A fragment from a row-major smem tile s[row][k] (k contiguous, leading dimension ld elements):
// rows r0..r0+15, contraction slice k0..k0+KStep-1.
template <typename T>
__device__ __forceinline__ void load_a(FragA<T, true>& f, const T* s, int ld, int r0, int k0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const T* p0 = s + (r0 + g) * ld + k0 + 2 * t;
  const T* p1 = p0 + 8 * ld;
  f.r[0] = *reinterpret_cast<const uint32_t*>(p0);
  f.r[1] = *reinterpret_cast<const uint32_t*>(p1);
  f.r[2] = *reinterpret_cast<const uint32_t*>(p0 + 8);
  f.r[3] = *reinterpret_cast<const uint32_t*>(p1 + 8);
}
template <typename T>
__device__ __forceinline__ void load_a(FragA<T, false>& f, const T* s, int ld, int r0, int k0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* p0 = reinterpret_cast<const float*>(s) + (r0 + g) * ld + k0 + t;
  const float* p1 = p0 + 8 * ld;
  split_t<T>(p0[0], f.hi[0], f.lo[0]);
  split_t<T>(p1[0], f.hi[1], f.lo[1]);
  split_t<T>(p0[4], f.hi[2], f.lo[2]);
  split_t<T>(p1[4], f.hi[3], f.lo[3]);
}

// B fragment, "NT": the smem tile is s[n][k] with k contiguous (C = A * s^T).
template <typename T>
__device__ __forceinline__ void load_b_nt(FragB<T, true>& f, const T* s, int ld, int n0, int k0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const T* p = s + (n0 + g) * ld + k0 + 2 * t;
  f.r[0] = *reinterpret_cast<const uint32_t*>(p);
  f.r[1] = *reinterpret_cast<const uint32_t*>(p + 8);
}
template <typename T>
__device__ __forceinline__ void load_b_nt(FragB<T, false>& f, const T* s, int ld, int n0, int k0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* p = reinterpret_cast<const float*>(s) + (n0 + g) * ld + k0 + t;
  split_t<T>(p[0], f.hi[0], f.lo[0]);
  split_t<T>(p[4], f.hi[1], f.lo[1]);
}

// B fragment, "NN": the smem tile is s[k][n] with n contiguous (C = A * s).
// 16-bit: slot pairs (2t,2t+1) and (2t+8,2t+9) are two consecutive rows of s.
// fp32: the A operand of these products comes straight from an accumulator tile whose
// columns (2t, 2t+1) sit in MMA k-slots (t, t+4) (see a_from_acc); the same permutation
// of the contraction index is applied here, so slot t reads row k0+2t and slot t+4 reads
// row k0+2t+1.
template <typename T>
__device__ __forceinline__ void load_b_nn(FragB<T, true>& f, const T* s, int ld, int k0, int n0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const unsigned short* p = reinterpret_cast<const unsigned short*>(s) + (k0 + 2 * t) * ld + n0 + g;
  f.r[0] = (uint32_t)p[0] | ((uint32_t)p[ld] << 16);
  f.r[1] = (uint32_t)p[8 * ld] | ((uint32_t)p[9 * ld] << 16);
}
template <typename T>
__device__ __forceinline__ void load_b_nn(FragB<T, false>& f, const T* s, int ld, int k0, int n0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const float* p = reinterpret_cast<const float*>(s) + (k0 + 2 * t) * ld + n0 + g;
  split_t<T>(p[0], f.hi[0], f.lo[0]);
  split_t<T>(p[ld], f.hi[1], f.lo[1]);
}

// A fragment taken from an accumulator-layout tile acc[n_tile][4] (16 rows x 8*n_tiles cols),
// contraction step kk (KStep columns starting at kk*KStep).
template <typename T>
__device__ __forceinline__ void a_from_acc(FragA<T, true>& f, const float (*acc)[4], int kk) {
  const float* c0 = acc[2 * kk];
  const float* c1 = acc[2 * kk + 1];
  f.r[0] = Elem<T>::pack(c0[0], c0[1]);
  f.r[1] = Elem<T>::pack(c0[2], c0[3]);
  f.r[2] = Elem<T>::pack(c1[0], c1[1]);
  f.r[3] = Elem<T>::pack(c1[2], c1[3]);
}
template <typename T>
__device__ __forceinline__ void a_from_acc(FragA<T, false>& f, const float (*acc)[4], int kk) {
  const float* c = acc[kk];
  split_t<T>(c[0], f.hi[0], f.lo[0]);  // slot t    <- column 2t,   row g
  split_t<T>(c[2], f.hi[1], f.lo[1]);  // slot t    <- column 2t,   row g+8
  split_t<T>(c[1], f.hi[2], f.lo[2]);  // slot t+4  <- column 2t+1, row g
  split_t<T>(c[3], f.hi[3], f.lo[3]);  // slot t+4  <- column 2t+1, row g+8
}

// ----------------------------------------------------------------------------------------------
// cp.async staging of a [ROWS][D] tile (rows row0.. of one head) into padded smem.
// Rows at or beyond L are zero-filled.
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc, int src_bytes) {
  uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gsrc), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// row_stride: elements between consecutive rows of the head in global memory (D for a row-major head; the row stride of
// a strided (batch, head, row) layout otherwise; the row itself is contiguous).
template <typename T, int ROWS, int D, int NTHREADS>
__device__ __forceinline__ void stage_tile(T* s, const T* head, int row0, int L, int tid, long long row_stride = D) {
  constexpr int LD = D + Elem<T>::kPad;
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int VPR = D / VEC;
  for (int idx = tid; idx < ROWS * VPR; idx += NTHREADS) {
    const int r = idx / VPR;
    const int c = (idx - r * VPR) * VEC;
    const int gr = row0 + r;
    const bool ok = gr < L;
    cp_async16(s + r * LD + c, head + (long long)(ok ? gr : 0) * row_stride + c, ok ? 16 : 0);
  }
}

// ----------------------------------------------------------------------------------------------
// Mask / bias accessor for one (batch, head).
// ----------------------------------------------------------------------------------------------
struct MaskView {
  int kind;
  int L;
  int kv_len;         // KVLEN: valid keys of this batch entry
  int bias_dtype;     // BIAS: jvpfa_dtype
  const void* base;   // BOOL / BIAS: pointer already offset to (b, h, 0, 0)
  long long si, sj;   // element strides along query / key

  __device__ __forceinline__ bool allowed(int i, int j) const {
    if (i >= L || j >= L) return false;
    switch (kind) {
      case JVPFA_MASK_CAUSAL:
        return j <= i;
      case JVPFA_MASK_KVLEN:
        return j < kv_len;
      case JVPFA_MASK_BOOL:
        return reinterpret_cast<const uint8_t*>(base)[i * si + j * sj] != 0;
      default:
        return true;
    }
  }
  // allowed() and bias() for the two neighbouring keys j, j + 1 (j even) of query i at once.  When the key
  // stride is 1 and the address allows it, the two mask bytes / bias elements come from one load.
  __device__ __forceinline__ void pair(int i, int j, bool ok[2], float b[2]) const {
    b[0] = b[1] = 0.f;
    if ((kind == JVPFA_MASK_BOOL || kind == JVPFA_MASK_BIAS) && sj == 1 && i < L && j + 1 < L) {
      const long long off = i * si + j;
      if (kind == JVPFA_MASK_BOOL) {
        const uint8_t* p = reinterpret_cast<const uint8_t*>(base) + off;
        if ((reinterpret_cast<uintptr_t>(p) & 1u) == 0) {
          const uint32_t w = *reinterpret_cast<const uint16_t*>(p);
          ok[0] = (w & 0xffu) != 0, ok[1] = (w >> 8) != 0;
          return;
        }
      } else if (bias_dtype == JVPFA_FP32) {
        const float* p = reinterpret_cast<const float*>(base) + off;
        if ((reinterpret_cast<uintptr_t>(p) & 7u) == 0) {
          const float2 v = *reinterpret_cast<const float2*>(p);
          ok[0] = ok[1] = true, b[0] = v.x, b[1] = v.y;
          return;
        }
      } else {
        const uint16_t* p = reinterpret_cast<const uint16_t*>(base) + off;
        if ((reinterpret_cast<uintptr_t>(p) & 3u) == 0) {
          const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
          ok[0] = ok[1] = true;
          if (bias_dtype == JVPFA_BF16) {
            b[0] = __uint_as_float(w << 16), b[1] = __uint_as_float(w & 0xffff0000u);
          } else {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
            b[0] = v.x, b[1] = v.y;
          }
          return;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      ok[e] = allowed(i, j + e);
      if (ok[e]) b[e] = bias(i, j + e);
    }
  }
  // Additive bias in natural units (0 unless kind == BIAS).  Only call for in-range (i, j).
  __device__ __forceinline__ float bias(int i, int j) const {
    if (kind != JVPFA_MASK_BIAS) return 0.f;
    const long long off = i * si + j * sj;
    if (bias_dtype == JVPFA_FP32) return reinterpret_cast<const float*>(base)[off];
    if (bias_dtype == JVPFA_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[off]);
    return __half2float(reinterpret_cast<const __half*>(base)[off]);
  }
};

__device__ __forceinline__ MaskView make_mask_view(const jvpfa_mask& m, int b, int h, int L) {
  MaskView v;
  v.kind = m.kind;
  v.L = L;
  v.kv_len = L;
  v.bias_dtype = m.bias_dtype;
  v.base = nullptr;
  v.si = m.stride[2];
  v.sj = m.stride[3];
  if (m.kind == JVPFA_MASK_KVLEN) {
    int n = m.kv_len[b];
    v.kv_len = n < 0 ? 0 : (n > L ? L : n);
  } else if (m.kind == JVPFA_MASK_BOOL) {
    v.base = reinterpret_cast<const uint8_t*>(m.ptr) + (long long)b * m.stride[0] + (long long)h * m.stride[1];
  } else if (m.kind == JVPFA_MASK_BIAS) {
    const long long off = (long long)b * m.stride[0] + (long long)h * m.stride[1];
    const int esz = (m.bias_dtype == JVPFA_FP32) ? 4 : 2;
    v.base = reinterpret_cast<const uint8_t*>(m.ptr) + off * esz;
  }
  return v;
}

// Reductions across the four lanes that share an accumulator row.
__device__ __forceinline__ float quad_max(float x) {
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
  x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
  return x;
}
__device__ __forceinline__ float quad_sum(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}

// Sums the register tiles x[ND][4] of the KG warps that share a row group into the kg = 0 warp, halving the number of
// parts in each step.  buf: (RG * KG / 2) * ND * 32 float4; ends (and begins) with nobody reading it.
template <int RG, int KG, int ND>
__device__ __forceinline__ void merge_parts(float4* buf, float (*x)[4], int rg, int kg, int lane) {
#pragma unroll
  for (int half = KG / 2; half > 0; half /= 2) {
    float4* p = buf + (size_t)((kg % half) * RG + rg) * ND * 32 + lane;
    if (kg >= half && kg < 2 * half) {
#pragma unroll
      for (int i = 0; i < ND; ++i) p[i * 32] = make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
    }
    __syncthreads();
    if (kg < half) {
#pragma unroll
      for (int i = 0; i < ND; ++i) {
        const float4 v = p[i * 32];
        x[i][0] += v.x, x[i][1] += v.y, x[i][2] += v.z, x[i][3] += v.w;
      }
    }
    __syncthreads();
  }
}

template <int N>
__device__ __forceinline__ void zero_acc(float (*x)[4]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    x[i][0] = 0.f;
    x[i][1] = 0.f;
    x[i][2] = 0.f;
    x[i][3] = 0.f;
  }
}

// Writes a warp's 16 x D accumulator strip (scaled) into a padded smem tile as T.
template <typename T, int D>
__device__ __forceinline__ void acc_to_smem(T* s, int ld, int r0, int lane, const float (*acc)[4], float scale) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int dt = 0; dt < D / 8; ++dt) {
    T* lo = s + (r0 + g) * ld + dt * 8 + 2 * t;
    T* hi = lo + 8 * ld;
    lo[0] = Elem<T>::from_float(acc[dt][0] * scale);
    lo[1] = Elem<T>::from_float(acc[dt][1] * scale);
    hi[0] = Elem<T>::from_float(acc[dt][2] * scale);
    hi[1] = Elem<T>::from_float(acc[dt][3] * scale);
  }
}

template <typename T, int ROWS, int D, int NTHREADS>
__device__ __forceinline__ void smem_tile_to_global(T* ghead, const T* s, int ld, int row0, int L, int tid) {
  constexpr int VEC = 16 / (int)sizeof(T);
  constexpr int VPR = D / VEC;
  for (int idx = tid; idx < ROWS * VPR; idx += NTHREADS) {
    const int r = idx / VPR, c = (idx - r * VPR) * VEC;
    const int row = row0 + r;
    if (row < L)
      *reinterpret_cast<uint4*>(ghead + (size_t)row * D + c) = *reinterpret_cast<const uint4*>(s + r * ld + c);
  }
}

// ---- Launches that follow one another ----------------------------------------------------------
// A kernel launched by launch_behind may be set up while the one before it on its stream still runs.  Every block of it begins with
// behind_previous: it waits until that one is complete, and all before it, and then lets the next one be set up.  So a kernel reads
// and writes what it likes behind that line, as after a plain launch, and only the launch itself is hidden, 1 to 2 us.  (Every
// block: else the kernel after it could start too early.)  fp16 B3 H12 L1330 D64 causal, forward and backward without tangents: 82.7 -> 76 us.
// pre_kernel is launched plainly: with it and the single-pass backward behind it both set up early that one took 210 us for 188
// (B4 H16 L2048 causal through tO), whatever the others did.
__device__ __forceinline__ void behind_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... Params, typename... Args>
cudaError_t launch_behind(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr, cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

// Raises a kernel's dynamic shared-memory limit once per device (the call costs about a microsecond of host time).
struct SmemOptIn {
  unsigned long long done = 0;  // bit per device; setting it twice does no harm
  bool ensure(const void* kernel, size_t bytes);
};

// The register-tiled kernels have two forms: a row group's loop split among several warps (fwd_generic.cu, bwd_generic.cu), and
// one warp for each 16 rows with little in registers (fwd_rows.cu, bwd_rows.cu).  The first fills the GPU from fewer rows, the
// second hides more latency once there are enough of them: n16 = 16-row tiles of the call.  Measured on a B200 at n16 = 32,
// 256, 512, 1008, 2048 and 8192 (split form / one warp form):
//   forward, O alone     16 bit D64 0.66 at 512, 1.15 at 2048   TF32 D64 0.83 at 1008, 1.29 at 2048   fp32 D64 0.97, 1.30
//   forward, tangents    16 bit D64 0.93 at 1008, 1.29 at 2048, D32 0.88 at 2048   TF32 D64 1.05, 1.24   fp32 D64 0.97, 1.04, D128 0.80
//   backward through O   16 bit D64 0.93 at 512, 1.36 at 1008   TF32 D64 0.98 at 512, 1.44 at 1008   fp32 D64 0.71, 1.16
//   backward, tangents   16 bit D64 0.78 at 512, 1.25 at 1008, D128 0.86   TF32 D32 1.18 at 1008, D64 0.89   fp32 D32 0.99, D64 0.57
// The lines lie between the sizes of either side, at four (backward) and eight (forward) 16-row tiles for each of the 148 SMs;
// TF32 at D = 128 gains least from the split (tangents 0.79 at 256, 1.08 at 512) and leaves it at two.  Variants of the second
// form that are never the better one are not compiled.
inline long long tiles16(int B, int H, int L) { return (long long)((L + 15) / 16) * B * H; }
template <typename T, int D>
constexpr bool kTf32AtD128 = !Elem<T>::k16 && !Elem<T>::kSplit && D == 128;
template <typename T, int D>
constexpr long long kFwdRowsFrom = kTf32AtD128<T, D> ? 2 * 148 : 8 * 148;
template <typename T, int D>
constexpr long long kBwdRowsFrom = kTf32AtD128<T, D> ? 2 * 148 : 4 * 148;
template <typename T, int D>
constexpr bool kFwdRowsDual = Elem<T>::k16 ? D > 32 : Elem<T>::kSplit ? D == 64 : true;
template <typename T, int D>
constexpr bool kBwdRowsDual = Elem<T>::k16 ? D <= 64 : !Elem<T>::kSplit && D == 32;

// Whether a part of a loop tile of the register-tiled kernels holds no true entry for the own tile, by the bitmaps of jvpfa_mask_tiles.  The tile is
// staged all the same and its products left out.  fp32 (and TF32) alone, in instances of their own (TILES): in those of other calls the test took
// registers, which cost most of them 1 to 3 % and TF32 at D = 64 through tO, which no longer fitted two CTAs on an SM, up to 1.4 times (B1 H8 L1000 275 /
// 366 us).  fp32, windows of a quarter of the length, us before / so, forward with tangents and backward through
// tO: B1 H2 L1410 D64 172 / 90 and 436 / 236, B2 H10 L1408 D32 390 / 211 and 1023 / 601, B1 H1 L704 D128
// 88 / 61 and 206 / 139.
inline bool with_tiles(const jvpfa_fwd_args& a) { return a.mask.kind == JVPFA_MASK_BOOL && a.mask_tile_live != nullptr; }
inline bool with_tiles(const jvpfa_bwd_args& a) {  // (both or neither)
  return a.mask.kind == JVPFA_MASK_BOOL && a.mask_tile_live != nullptr && a.mask_tile_live_t != nullptr;
}
__device__ __forceinline__ long long bitmap_head(const jvpfa_mask& m, int b, int h, int H) {  // (a dimension that broadcasts has one entry)
  return (m.stride[0] ? (long long)b * (m.stride[1] ? H : 1) : 0) + (m.stride[1] ? h : 0);
}
__device__ __forceinline__ bool no_bit(const void* bitmap, long long word, int from, int to) {
  const unsigned long long* w = reinterpret_cast<const unsigned long long*>(bitmap) + word;
  bool any = false;
  for (int b = from; b <= to; ++b) any = any || ((__ldg(w + (b >> 6)) >> (b & 63)) & 1ull);
  return !any;
}
// Own queries from m0 on (of one 128-query tile) and keys [n0, n1).
template <typename Args>
__device__ __forceinline__ bool dead_keys(const Args& a, int b, int h, int m0, int n0, int n1) {
  const long long head = bitmap_head(a.mask, b, h, a.H);
  return no_bit(a.mask_tile_live, (a.mask.stride[2] ? head * ((a.L + 127) / 128) + m0 / 128 : head) * (((a.L + 63) / 64 + 63) / 64), n0 >> 6, (n1 - 1) >> 6);
}
// Own keys from n0 on (of one 128-key tile) and queries [m0, m1).
__device__ __forceinline__ bool dead_queries(const jvpfa_bwd_args& a, int b, int h, int n0, int m0, int m1) {
  const bool rows = a.mask.stride[2] != 0;
  const int n_t128 = (a.L + 127) / 128;
  return no_bit(a.mask_tile_live_t, (bitmap_head(a.mask, b, h, a.H) * n_t128 + n0 / 128) * (rows ? (n_t128 + 63) / 64 : 1), rows ? m0 >> 7 : 0,
                rows ? (m1 - 1) >> 7 : 0);
}

// 16-row groups of a CTA of the fp32 register-tiled kernels with tangents, 1, 2 or 4 (and 8, 4 or 2 parts of the loop side).  64 rows share every tile
// that is brought in, and 16 take cost1 percent of their time for a row, 32 cost2, but a launch takes rounds of as many CTAs as 148 SMs hold: fit of
// each kind on one, of which each but the first adds `beside` percent of its time.  Causal: half the work, evened out, and `tail` percent of a CTA's.
// `fit` is what registers and shared memory allow (-Xptxas -v: D >= 64 takes 129 to 255 registers at 256 threads, but for TF32's backward in 32
// rows; D = 32 at most 128, and 80 in TF32's backward in 32 rows), the rest a fit to 2896 draws on a B200 (B*H of 1 to 300, L of 66 to 2400, 60 to 1500
// groups, forward and backward through tO), in each of which all three kinds were timed.  Slower than the best of the three by so much in the mean, of
// draws where they differ, by the number of rows alone (64 from 592 groups on, 32 from 296) / as if one CTA of any filled an SM, with cost1 of 145
// and 132 / by this rule: fp32 forward D = 32 6.4 / 3.4 / 1.5 %, 64 4.7 / 0.7 / 0.7, 128 4.7 / 1.0 / 0.6, backward 7.1 / 2.3 / 1.0, 8.0 / 3.0 / 0.8,
// 7.7 / 1.5 / 0.8; TF32 forward 4.0 / 6.0 / 1.5, 8.1 / 5.4 / 1.1, 7.9 / 0.8 / 0.3, backward 3.3 / 4.6 / 0.7, 10.4 / 12.6 / 0.5, 6.7 / 6.0 / 0.4.  us by 16 /
// 32 / 64 rows: TF32 backward D = 64 B1 H241 L92 causal 146 / 72 / 99, forward D = 32 B3 H41 L66 19 / 15 / 11; fp32 forward D = 32 B1 H131 L76 25 / 19 / 19,
// backward D = 64 B1 H282 L72 218 / 157 / 187.
// Without tangents two CTAs of short row tiles fit an SM, and the number of rows does decide (B1 H2 L1410, 16 / 32 rows: 84 / 109).
struct RowGroups {
  int fit[3];
  int cost1, cost2, beside, tail;
};
template <typename T, int D>
constexpr RowGroups kFwdRowGroups = Elem<T>::kSplit ? (D == 32   ? RowGroups{{2, 2, 2}, 174, 111, 25, 217}
                                                       : D == 64 ? RowGroups{{1, 1, 1}, 179, 110, 0, 180}
                                                                 : RowGroups{{1, 1, 1}, 175, 102, 0, 225})
                                                    : (D == 32   ? RowGroups{{2, 2, 2}, 194, 137, 14, 60}
                                                       : D == 64 ? RowGroups{{1, 1, 1}, 219, 151, 0, 75}
                                                                 : RowGroups{{1, 1, 1}, 146, 103, 0, 63});
template <typename T, int D>
constexpr RowGroups kBwdRowGroups = Elem<T>::kSplit ? (D == 32   ? RowGroups{{2, 2, 2}, 134, 111, 56, 97}
                                                       : D == 64 ? RowGroups{{1, 1, 1}, 158, 108, 0, 143}
                                                                 : RowGroups{{1, 1, 1}, 135, 114, 0, 88})
                                                    : (D == 32   ? RowGroups{{2, 3, 2}, 153, 147, 18, 32}
                                                       : D == 64 ? RowGroups{{1, 2, 1}, 216, 132, 48, 244}
                                                                 : RowGroups{{1, 1, 1}, 222, 150, 0, 89});
inline int row_groups(int B, int H, int L, bool tangents, bool causal, const RowGroups& kinds) {
  const long long rows16 = tiles16(B, H, L);
  if (!tangents) return rows16 < 2 * 148 ? 1 : rows16 < 4 * 148 ? 2 : 4;
  const long long BH = (long long)B * H;
  auto time = [&](int rg, int fit, int cost) {
    const long long ctas = BH * ((L + 16 * rg - 1) / (16 * rg)), deep = (ctas + 147) / 148, last = deep % fit;
    const int full = 100 + (fit - 1) * kinds.beside;
    const double t = causal ? (double)(ctas * full) / (2 * 148 * fit) + kinds.tail
                            : (double)(deep / fit * full + (last ? 100 + (last - 1) * kinds.beside : 0));
    return t * rg * cost;
  };
  const double one = time(1, kinds.fit[0], kinds.cost1), two = time(2, kinds.fit[1], kinds.cost2), four = time(4, kinds.fit[2], 100);
  return one <= two && one <= four ? 1 : two <= four ? 2 : 4;
}

// Host-side launch helpers implemented by each kernel translation unit.
int launch_fwd_generic(const jvpfa_fwd_args& a, cudaStream_t stream);
int launch_fwd_rows(const jvpfa_fwd_args& a, cudaStream_t stream);
int launch_bwd_rows(const jvpfa_bwd_args& a, cudaStream_t stream);
int launch_pre(const jvpfa_pre_args& a, cudaStream_t stream);
int launch_bwd_generic(const jvpfa_bwd_args& a, cudaStream_t stream);
int launch_mask_check(const jvpfa_mask_check_args& a, cudaStream_t stream);
int launch_mask_tiles(const jvpfa_mask_tiles_args& a, cudaStream_t stream);
int launch_pad_bias(const jvpfa_pad_bias_args& a, cudaStream_t stream);
int launch_fwd_tc5(const jvpfa_fwd_args& a, cudaStream_t stream);
bool fwd_tc5_eligible(const jvpfa_fwd_args& a);
bool tc5_head_dim(int D, int L);
bool tc5_mask_layout(const jvpfa_mask& m, int dtype, int L);
int tc5_read_status(int* out, int clear);
int tc5_status_peek();
int tc5_inject_status(int code);
int* tc5_status_device_ptr();
int launch_bwd_tc5(const jvpfa_bwd_args& a, cudaStream_t stream);
int launch_bwd_tc5_d64(const jvpfa_bwd_args& a, cudaStream_t stream);
int launch_bwd_tc5_fused64(const jvpfa_bwd_args& a, cudaStream_t stream);
bool bwd_tc5_fused64_eligible(const jvpfa_bwd_args& a);
long long bwd_fused64_workspace(const jvpfa_bwd_args& a);
long long fwd_pair64_workspace(const jvpfa_fwd_args& a);
int launch_fwd_tc5_pair64(const jvpfa_fwd_args& a, cudaStream_t stream);
int launch_fwd_tc5_pipe128(const jvpfa_fwd_args& a, cudaStream_t stream);
bool bwd_tc5_pipe128_eligible(const jvpfa_bwd_args& a);
int launch_bwd_tc5_pipe128(const jvpfa_bwd_args& a, cudaStream_t stream);
bool bwd_tc5_eligible(const jvpfa_bwd_args& a);
long long fwd_f32_tc5_workspace(const jvpfa_fwd_args& a);
bool fwd_f32_tc5_eligible(const jvpfa_fwd_args& a);
int launch_fwd_f32_tc5(const jvpfa_fwd_args& a, cudaStream_t stream);
long long bwd_f32_tc5_workspace(const jvpfa_bwd_args& a);
bool bwd_f32_tc5_eligible(const jvpfa_bwd_args& a);
int launch_bwd_f32_tc5(const jvpfa_bwd_args& a, cudaStream_t stream);
void set_last_cuda_error(cudaError_t e, const char* where);
int check_pre_request(const jvpfa_pre_args* a);
int check_bwd_request(const jvpfa_bwd_args* a);

}  // namespace jvpfa
