// One pass over a user mask that answers what upstream asks of it before a forward
// (jvp_flash_attention/jvp_attention.py:2438-2457): does every head of a boolean mask keep at least
// one entry, does a floating-point mask contain inf or NaN, does every head of it have at least one
// entry other than the masking constant -100.  Upstream answers with four eager reductions over the
// whole mask and a host synchronisation after each; here one HBM-bound kernel writes one int32 per
// head plus one "bad value" word, which the caller reads back once.
//
// Work split: blockIdx.y = head of the mask (its own batch x head extents: broadcast dimensions
// count once), blockIdx.x = a slice of that head's rows.  A row is read as 16-byte vectors when its
// key stride is 1 and it starts on a 16-byte boundary, element by element otherwise.
#include "common.cuh"

namespace jvpfa {

namespace {

constexpr int kCheckThreads = 256;

// bit 0: the element counts as "live" (true / not the masking constant -100); bit 1: inf; bit 2: NaN
__device__ __forceinline__ uint32_t classify_bits(uint32_t x, uint32_t mask_const, uint32_t exp_mask, uint32_t man_mask) {
  uint32_t r = x != mask_const ? 1u : 0u;
  if ((x & exp_mask) == exp_mask) r |= (x & man_mask) ? 4u : 2u;
  return r;
}
template <int KIND_DTYPE>
__device__ __forceinline__ uint32_t classify16(uint32_t h) {
  if constexpr (KIND_DTYPE == JVPFA_BF16)
    return classify_bits(h & 0xffffu, 0xC2C8u, 0x7f80u, 0x007fu);
  else
    return classify_bits(h & 0xffffu, 0xD640u, 0x7c00u, 0x03ffu);
}
__device__ __forceinline__ uint32_t classify32(uint32_t w) { return classify_bits(w, 0xC2C80000u, 0x7f800000u, 0x007fffffu); }

// MODE 0: uint8 mask; 1: bf16; 2: fp16; 3: fp32
template <int MODE>
__device__ __forceinline__ uint32_t classify_word(uint32_t w) {
  if constexpr (MODE == 0) return w != 0u ? 1u : 0u;
  if constexpr (MODE == 1) return classify16<JVPFA_BF16>(w) | classify16<JVPFA_BF16>(w >> 16);
  if constexpr (MODE == 2) return classify16<JVPFA_FP16>(w) | classify16<JVPFA_FP16>(w >> 16);
  return classify32(w);
}

template <int MODE>
__device__ __forceinline__ uint32_t classify_elem(const unsigned char* p) {
  if constexpr (MODE == 0) return *p != 0 ? 1u : 0u;
  if constexpr (MODE == 1) return classify16<JVPFA_BF16>(*reinterpret_cast<const uint16_t*>(p));
  if constexpr (MODE == 2) return classify16<JVPFA_FP16>(*reinterpret_cast<const uint16_t*>(p));
  return classify32(*reinterpret_cast<const uint32_t*>(p));
}

template <int MODE>
__global__ void __launch_bounds__(kCheckThreads) mask_check_kernel(const jvpfa_mask m, int n_h, int n_rows, int L,
                                                                   int rows_per_cta, int32_t* out) {
  constexpr int ESZ = MODE == 0 ? 1 : (MODE == 3 ? 4 : 2);
  constexpr int EPV = 16 / ESZ;  // elements per 16-byte vector
  const int head = blockIdx.y;
  const int b = head / n_h, h = head - b * n_h;
  const int r0 = blockIdx.x * rows_per_cta;
  const int r1 = min(n_rows, r0 + rows_per_cta);
  const unsigned char* base =
      reinterpret_cast<const unsigned char*>(m.ptr) + ((long long)b * m.stride[0] + (long long)h * m.stride[1]) * ESZ;
  const long long row_bytes = m.stride[2] * ESZ;
  const bool vec = m.stride[3] == 1 && (L % EPV) == 0 && (reinterpret_cast<uintptr_t>(base) & 15u) == 0 &&
                   (row_bytes & 15) == 0;
  uint32_t acc = 0;
  auto take = [&](const uint4 x) {
    acc |= classify_word<MODE>(x.x) | classify_word<MODE>(x.y) | classify_word<MODE>(x.z) | classify_word<MODE>(x.w);
  };
  if (vec) {
    const int vpr = L / EPV;
    if (row_bytes == (long long)L * ESZ) {  // the slice is one contiguous range
      const uint4* p = reinterpret_cast<const uint4*>(base + (long long)r0 * row_bytes);
      const int total = (r1 - r0) * vpr;
#pragma unroll 8
      for (int idx = threadIdx.x; idx < total; idx += kCheckThreads) take(__ldg(p + idx));
    } else {
      for (int r = r0; r < r1; ++r) {
        const uint4* p = reinterpret_cast<const uint4*>(base + (long long)r * row_bytes);
#pragma unroll 4
        for (int c = threadIdx.x; c < vpr; c += kCheckThreads) take(__ldg(p + c));
      }
    }
  } else {
    for (int r = r0; r < r1; ++r) {
      const unsigned char* p = base + (long long)r * row_bytes;
      for (int c = threadIdx.x; c < L; c += kCheckThreads) acc |= classify_elem<MODE>(p + (long long)c * m.stride[3] * ESZ);
    }
  }
  const int live = __syncthreads_or((int)(acc & 1u));
  const int inf = __syncthreads_or((int)(acc & 2u));
  const int nan = __syncthreads_or((int)(acc & 4u));
  if (threadIdx.x == 0) {
    if (live) out[1 + head] = 1;  // every writer stores the same value
    if (inf || nan) atomicOr(out, (inf ? 1 : 0) | (nan ? 2 : 0));
  }
}

// Summaries of a boolean mask: one bit per 128 x 64 tile with a true entry (both orientations), and the mask itself as
// one bit per entry, by rows and transposed.  The attention kernels then read 8 bytes of a mask row per 64-key tile
// instead of 64, and where a thread owns a key one word instead of 32 single bytes, each from another row.
//
// HBM bound (1 byte read and 1/4 byte written per entry).  A warp takes 32 rows x 512 keys: lane l reads bytes
// [16 l, 16 l + 16) of each row, keeps them as 16 bits, and builds its 16 transposed words bit by bit on the way; the
// CTA's eight warps (256 rows) pass those through shared memory so that they leave as 32-byte pieces.
// With the packed mask, B2 H12 L2048 D64 and nine tenths random False: forward with tangents 168 -> 151 us, backward
// through tO 239 -> 186 us.
constexpr int kPackRows = 256, kPackKeys = 512;

__device__ __forceinline__ uint32_t nonzero_bits(uint32_t w) {  // bytes -> four bits
  return (((__vcmpne4(w, 0u) & 0x01010101u) * 0x01020408u) >> 24) & 0xfu;
}

__global__ void __launch_bounds__(256) mask_pack_kernel(const jvpfa_mask m, int n_h, int n_rows, int L, int n_qt, int n_words,
                                                        unsigned char* tile_live, int32_t* head_live,
                                                        unsigned long long* tile_live_t, int n_kt128, int n_words_t,
                                                        uint32_t* bits, uint32_t* bits_t) {
  __shared__ unsigned int s_tiles[2];                       // of the CTA's two 128-row tiles
  __shared__ uint32_t s_t[kPackKeys * 8 + kPackKeys / 16];  // [key][warp], one word of padding per 16 keys
  const int head = blockIdx.z, kg = blockIdx.x;             // kg: group of eight key tiles
  const int b = head / n_h, h = head - b * n_h;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(m.ptr) + (long long)b * m.stride[0] + (long long)h * m.stride[1];
  const long long rs = m.stride[2], ks = m.stride[3];
  if (threadIdx.x < 2) s_tiles[threadIdx.x] = 0u;
  const int col = kg * kPackKeys + lane * 16;
  const int row0 = blockIdx.y * kPackRows + warp * 32;
  const bool vec = ks == 1 && (rs & 15) == 0 && (reinterpret_cast<uintptr_t>(base) & 15u) == 0 && col + 16 <= L;
  const int w_rows = ((L + 63) / 64) * 2;  // words of a row
  uint32_t t[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) t[j] = 0u;
  uint32_t any = 0u;
#pragma unroll 8
  for (int r = 31; r >= 0; --r) {  // downwards: the first row ends up in bit 0
    const int row = row0 + r;
    uint32_t x = 0u;
    if (row < n_rows && col < L) {
      const unsigned char* p = base + (long long)row * rs + (long long)col * ks;
      if (vec) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        x = nonzero_bits(v.x) | nonzero_bits(v.y) << 4 | nonzero_bits(v.z) << 8 | nonzero_bits(v.w) << 12;
      } else {
        const int n = min(16, L - col);
        for (int j = 0; j < n; ++j) x |= (p[j * ks] != 0 ? 1u : 0u) << j;
      }
    }
    any |= x;
#pragma unroll
    for (int j = 0; j < 16; ++j) t[j] = (t[j] << 1) | ((x >> j) & 1u);
    const uint32_t other = __shfl_xor_sync(0xffffffffu, x, 1);
    const int word = kg * (kPackKeys / 32) + (lane >> 1);
    if (bits != nullptr && (lane & 1) == 0 && row < n_rows && word < w_rows)
      bits[((long long)head * n_rows + row) * w_rows + word] = x | other << 16;
  }
  const unsigned int vote = __ballot_sync(0xffffffffu, any != 0u);  // bit l: lane l saw a true entry
  __syncthreads();
  if (lane == 0 && vote != 0u) {
    unsigned int tiles = 0u;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (vote & (0xfu << (4 * k))) tiles |= 1u << k;
    atomicOr(&s_tiles[warp >> 2], tiles);
  }
  if (bits_t != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) s_t[(lane * 16 + j) * 8 + warp + lane] = t[j];
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_tiles[threadIdx.x] != 0u && tile_live != nullptr) {
    const unsigned int tiles = s_tiles[threadIdx.x];
    const int qt = blockIdx.y * 2 + threadIdx.x;
    // byte kg of the entry's words (little endian: byte k of a word holds its bits 8k .. 8k+7)
    tile_live[((long long)head * n_qt + qt) * n_words * 8 + kg] = (unsigned char)tiles;
    if (head_live) {
      head_live[head] = 1;
      atomicAdd(head_live + gridDim.z, __popc(tiles));  // live tiles of the whole mask
    }
    if (tile_live_t) {  // the transposed summary: per 128-key tile, one bit per 128-query tile
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if ((tiles >> (2 * j)) & 3u)
          atomicOr(tile_live_t + ((long long)head * n_kt128 + 4 * kg + j) * n_words_t + (qt >> 6), 1ull << (qt & 63));
    }
  }
  if (bits_t != nullptr) {
    for (int k = threadIdx.x; k < kPackKeys; k += 256) {
      const int key = kg * kPackKeys + k;
      if (key >= L) break;
      const uint32_t* src = s_t + k * 8 + (k >> 4);
      if (n_rows == 1) {  // one row for every query: all bits of the key's only word alike
        bits_t[(long long)head * L + key] = (src[0] & 1u) ? ~0u : 0u;
        continue;
      }
      const int w_cols = ((n_rows + 63) / 64) * 2, w0 = blockIdx.y * (kPackRows / 32);
      uint2* dst = reinterpret_cast<uint2*>(bits_t + ((long long)head * L + key) * w_cols + w0);
#pragma unroll
      for (int w = 0; w < 4; ++w)
        if (w0 + 2 * w < w_cols) dst[w] = make_uint2(src[2 * w], src[2 * w + 1]);
    }
  }
}

}  // namespace

int launch_mask_tiles(const jvpfa_mask_tiles_args& a, cudaStream_t stream) {
  const int n_kt = (a.L + 63) / 64;
  const int n_words = (n_kt + 63) / 64;
  const int n_qt = a.n_rows == 1 ? 1 : (a.L + 127) / 128;
  const dim3 grid((unsigned)((n_kt + 7) / 8), (unsigned)((a.n_rows + kPackRows - 1) / kPackRows), (unsigned)(a.n_b * a.n_h));
  const int n_kt128 = (a.L + 127) / 128;
  const int n_words_t = (n_qt + 63) / 64;
  mask_pack_kernel<<<grid, 256, 0, stream>>>(a.mask, a.n_h, a.n_rows, a.L, n_qt, n_words,
                                             reinterpret_cast<unsigned char*>(a.tile_live), a.head_live,
                                             reinterpret_cast<unsigned long long*>(a.tile_live_t), n_kt128, n_words_t,
                                             reinterpret_cast<uint32_t*>(a.bits), reinterpret_cast<uint32_t*>(a.bits_t));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch mask_pack");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

int launch_mask_check(const jvpfa_mask_check_args& a, cudaStream_t stream) {
  const int n_heads = a.n_b * a.n_h;
  // about 32 KiB of mask per CTA (eight 16-byte loads per thread), at least one row: a 100 MB mask gives
  // some 3000 CTAs, enough loads in flight to run at HBM speed
  const long long row_bytes = (long long)a.L * (a.mask.kind == JVPFA_MASK_BOOL ? 1 : (a.mask.bias_dtype == JVPFA_FP32 ? 4 : 2));
  long long rpc = (32ll << 10) / row_bytes;
  if (rpc < 1) rpc = 1;
  if (rpc > a.n_rows) rpc = a.n_rows;
  const dim3 grid((unsigned)((a.n_rows + rpc - 1) / rpc), (unsigned)n_heads);
  if (a.mask.kind == JVPFA_MASK_BOOL)
    mask_check_kernel<0><<<grid, kCheckThreads, 0, stream>>>(a.mask, a.n_h, a.n_rows, a.L, (int)rpc, a.out);
  else if (a.mask.bias_dtype == JVPFA_BF16)
    mask_check_kernel<1><<<grid, kCheckThreads, 0, stream>>>(a.mask, a.n_h, a.n_rows, a.L, (int)rpc, a.out);
  else if (a.mask.bias_dtype == JVPFA_FP16)
    mask_check_kernel<2><<<grid, kCheckThreads, 0, stream>>>(a.mask, a.n_h, a.n_rows, a.L, (int)rpc, a.out);
  else
    mask_check_kernel<3><<<grid, kCheckThreads, 0, stream>>>(a.mask, a.n_h, a.n_rows, a.L, (int)rpc, a.out);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch mask_check");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

}  // namespace jvpfa
