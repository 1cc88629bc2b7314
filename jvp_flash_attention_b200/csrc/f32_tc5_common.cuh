// fp32 on the 16-bit tensor cores, without loss: what the kernels of fwd_f32_tc5.cu share.
//
// An fp32 number x is the sum of three bf16 numbers, hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid (24 significant bits
// are 8 + 8 + 8, the differences are exact), and bf16 has fp32's range of exponents, so every entry keeps its precision
// whatever else its row or column holds.  A product is the six MMAs hi*hi, hi*mid, mid*hi, mid*mid, hi*lo, lo*hi; what is left
// out (mid*lo, lo*mid, lo*lo) is at most 2^-24 of it, since |mid| <= 2^-8 and |lo| <= 2^-17 of the leading bit (above 2^-26 for
// 2.8 % of uniform pairs).  Of entries below 2^-109 bf16 no longer holds all of the lo part.
//
// The inputs are split once per call into a caller-owned workspace: three row-major (B*H, L, D) planes of bf16 per tensor,
// all of them one tensor map (D, L, B*H, planes).
#pragma once

#include "tc5_common.cuh"

namespace jvpfa {
namespace tc5 {

constexpr int kF32MaxSlots = 6;
constexpr int kSplitBlock = 256 * 8;  // elements that a block of the splitting pass takes

// Beside the status word: a wait of an fp32 kernel gave up.  Only this ends a later one on entry: an fp32 call that is queued, or
// replayed, behind a 16-bit launch that gave up is computed, as on the register-tiled kernels.
constexpr int kF32GaveUp = 1;

struct SplitArgs {
  const float* src[kF32MaxSlots];
  long long st[kF32MaxSlots][3];  // batch, head, row strides in elements
  __nv_bfloat16* dst;             // [slot][part][B*H][L][D]
  long long plane;                // B*H*L*D
  int H, L, D;
  // Key padding: what `padded` (a bit per slot) holds of keys that no query attends is written as zeros.  A tile of 64 keys goes
  // into the products whole, and an Inf or a NaN there would reach every row through its probability of 0.
  const int32_t* kv_len;
  unsigned padded;
  // Causal: what is not finite in the slots of `clean` is written as zero, for the same reason (rows of a query tile that end before
  // the key).  `found` (or null): which blocks of kSplitBlock elements of those slots, one after another, hold such an entry; the
  // kernel then looks at the entries themselves for the rows that attend them.
  unsigned clean;
  uint32_t* found;
  void set(int slot, const void* p, const int64_t* in_stride) {  // in_stride all zero or null: row-major
    src[slot] = static_cast<const float*>(p);
    const bool strided = in_stride && (in_stride[0] | in_stride[1] | in_stride[2]) != 0;
    st[slot][0] = strided ? in_stride[0] : (long long)H * L * D;
    st[slot][1] = strided ? in_stride[1] : (long long)L * D;
    st[slot][2] = strided ? in_stride[2] : D;
  }
};

// One value as three bf16 parts.  A value that rounds beyond bf16's range is cut instead; Inf and NaN make all that they enter NaN.
__device__ __forceinline__ void split3(float x, float& h, float& m, float& l) {
  uint32_t hb = __float_as_uint(__bfloat162float(__float2bfloat16_rn(x)));
  if ((hb & 0x7fffffffu) == 0x7f800000u) hb = __float_as_uint(x) & 0xffff0000u;
  h = __uint_as_float(hb);
  const float r = x - h;
  m = __bfloat162float(__float2bfloat16_rn(r));
  l = r - m;
}
// Two values, packed: the form in which they are stored or handed to the tensor cores.
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ void split3_pair(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(a, b);
  const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
  m = pack_bf16(ra, rb);
  l = pack_bf16(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xffff0000u));
}

// A score in base-2 units, as every kernel rounds it: what the backward subtracts lse from is what the forward made lse of.  (A
// product that goes unrounded into the subtraction, as the compiler would have it, is off by up to half a unit of the score: at
// |S| of 50 the probability of a row's only key came out 1 + 1e-6.)
template <int MK>
__device__ __forceinline__ float f32_score(float s, float scale_log2, float bias) {
  const float v = __fmul_rn(s, scale_log2);
  return MK == 2 ? __fmaf_rn(bias, kLog2e, v) : v;
}

// What a thread reads of the mask: 32 neighbouring keys of its query row i at a time.
// MK: 0 = none / causal / key padding; 1 = boolean mask (bits, or bytes of any strides); 2 = additive bias (any type and
// strides).
template <int MK>
struct F32RowMask {
  MaskView mv;
  const unsigned char* row;
  const uint32_t* bits;
  int L, i, esz;
  bool vec;  // the row can be read 16 bytes at a time

  __device__ __forceinline__ F32RowMask(const jvpfa_mask& m, const void* mask_bits, int b, int h, int H, int i_, int L_)
      : mv(make_mask_view(m, b, h, L_)), row(nullptr), bits(nullptr), L(L_), i(min(i_, L_ - 1)), esz(1), vec(false) {
    if constexpr (MK != 0) {
      if (MK == 2) esz = m.bias_dtype == JVPFA_FP32 ? 4 : 2;
      row = reinterpret_cast<const unsigned char*>(mv.base) + (long long)i * mv.si * esz;
      vec = mv.sj == 1 && (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
      if (MK == 1 && mask_bits != nullptr) bits = mask_bit_row(mask_bits, m, mask_head(m, b, h, H), i, L);
    }
  }
  // Keys n0 .. n0 + 31: a bit for each that the mask lets the row attend, of those in `live`; the bias.
  __device__ __forceinline__ uint32_t fetch(int n0, uint32_t live, float* bias) const {
    if constexpr (MK == 1) {
      uint32_t r = 0u;
      if (bits != nullptr) {
        r = n0 < L ? ldg_nc_u32(bits + (n0 >> 5)) : 0u;
      } else if (vec && n0 + 32 <= L) {
        const uint4 r0 = ldg_nc_v4(row + n0), r1 = ldg_nc_v4(row + n0 + 16);
        r = bits_of_bytes(r0.x) | bits_of_bytes(r0.y) << 4 | bits_of_bytes(r0.z) << 8 | bits_of_bytes(r0.w) << 12 |
            bits_of_bytes(r1.x) << 16 | bits_of_bytes(r1.y) << 20 | bits_of_bytes(r1.z) << 24 | bits_of_bytes(r1.w) << 28;
      } else {
#pragma unroll 8
        for (int c = 0; c < 32; ++c) r |= (ldg_nc_u8(row + (long long)min(n0 + c, L - 1) * mv.sj) != 0u ? 1u : 0u) << c;
      }
      live &= r;
    }
    if constexpr (MK == 2) {
      // (the piece of two 64-key tiles on is brought into L2 meanwhile: a row's pieces lie in DRAM pages of their own)
      if (mv.sj == 1 && n0 + 128 < L) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (size_t)(n0 + 128) * esz));
      if (vec && n0 + 32 <= L && esz == 4) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 r = ldg_nc_v4(row + (size_t)(n0 + 4 * c) * 4);
          bias[4 * c] = __uint_as_float(r.x), bias[4 * c + 1] = __uint_as_float(r.y);
          bias[4 * c + 2] = __uint_as_float(r.z), bias[4 * c + 3] = __uint_as_float(r.w);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) bias[c] = mv.bias(i, min(n0 + c, L - 1));
      }
    }
    return live;
  }
};

// Whether a call has rows enough for these kernels, which work on 128-row tiles and split their inputs first, not to be slower than
// the register-tiled ones, which fill the GPU from fewer.  n16: 16-row tiles of the call.  Measured on a B200, us of the device,
// register-tiled / here: O alone, with tangents, O and its three gradients; 64-row sequences (one tile, half of it empty) lose.
//   D = 64   L66  n16 385 16/16 31/25 53/49    bias 18/18 31/27 54/63   ragged boolean 18/29 33/37 55/74
//            L96  n16 384 16/18 31/27 55/51    bias 18/23 33/29 57/68   n16 672 bias 29/25 49/33 100/72
//            L130 n16 387 25/20 45/31 80/59    bias 25/25 45/33 79/76   ragged boolean 25/31 49/43 82/84, n16 774 43/41 72/61 145/121
//            L192 n16 384 27/20 51/33 94/57    bias 29/22 55/33 94/70   L512 n16 256 34/30 71/46, bias 36/42 74/65
//   D = 128  L66  n16 320 25/23 49/39 90/82    causal 25/23 41/39 78/82  bias 25/23 49/41 90/92, ragged boolean 25/33 51/57 92/106
//            L96  n16 324 25/23 51/41 96/86    causal 23/22 41/41 80/88  bias 27/27 53/45 96/100, n16 642 43/31 86/53 176/111
//            L112 n16 322 31/23 61/43 115/90   causal 29/23 47/43 96/90  bias 29/25 61/45 115/100
//   D = 32   L192 n16 1032 22/29 41/43 84/86   causal 25/27 41/39 82/76  n16 4104 53/61 119/104 207/203  (64-row tiles fit, 128 do not)
//            L200 n16 1027 35/31 66/47 119/96  bias 37/39 68/55 147/123; L208 n16 1027 bias 37/41, n16 1547 57/45
//            L256 n16 1024 29/23 51/33 106/61  bias 33/27 55/37 150/80
// Far above the lines nothing loses more than 3 % (D64 n16 12288: L66 244/188 610/330 917/631, L96 with bias 223/231 547/360
// 1059/727).  Below them long sequences gain as well (D = 128 n16 256, L2048: 249/101 469/249), short ones do not.
// `by_element`: a bias, and a boolean mask that is packed first because its rows are not whole 16-byte pieces.
inline bool f32_rows_enough(const jvpfa_mask& m, int B, int H, int L, int D) {
  const long long n16 = tiles16(B, H, L);
  const bool by_element =
      m.kind == JVPFA_MASK_BIAS || (m.kind == JVPFA_MASK_BOOL && ((L & 15) != 0 || !tc5_mask_layout(m, JVPFA_FP32, L)));
  if (D == 128) return L > 64 && n16 >= (L <= 96 && (by_element || m.kind == JVPFA_MASK_CAUSAL) ? 576 : 320);
  if (D == 64) return L > 64 && n16 >= (L < 192 && by_element ? 640 : 384);
  return L > 192 && n16 >= (L < 224 && by_element ? 1280 : 1024);
}

// Host: the splitting launch, and the tensor map of its result (boxes of 64 columns x 64 rows of one plane).
int launch_split3(const SplitArgs& s, int slots, cudaStream_t stream);
bool encode_map_parts(CUtensorMap* m, const void* ptr, int D, int L, int BH, int planes);

}  // namespace tc5
}  // namespace jvpfa
