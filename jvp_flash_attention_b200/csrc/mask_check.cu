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
// HBM bound (1 byte read and 1/4 byte written per entry), if enough of it is in flight: a warp takes 32 rows x 256 keys and
// a lane asks for its 8 bytes of all 32 rows at once.  Four lanes put a row's word together; eight rows at a time are
// transposed as 8 x 8 bits, and the CTA's eight warps (256 rows) pass the transposed words through shared memory so that
// they leave as 32-byte pieces.  B2 H12 L2048 (100 MB) 32 us, 36 where other kernels' lines leave L2 meanwhile; one head of L4096
// (17 MB) 8 us; 16 bytes of up to eight rows at a time and a transposition bit by bit took 60 and 25 us.
// With the packed mask, B2 H12 L2048 D64 and nine tenths random False: forward with tangents 140 -> 86 us, backward
// through tO 221 -> 142 us.
constexpr int kPackRows = 256, kPackKeys = 256;

__device__ __forceinline__ uint32_t nonzero_bits(uint32_t w) {  // bytes -> four bits
  const uint32_t top = (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;
  return (top * 0x00204081u) >> 28;  // bits 7, 15, 23, 31 -> 28 .. 31
}

// 8 x 8 bits, byte r of (lo, hi) = row r, transposed in place (H. S. Warren, "Hacker's Delight", 7-3).
__device__ __forceinline__ void transpose8(uint32_t& lo, uint32_t& hi) {
  uint32_t t = (lo ^ (lo >> 7)) & 0x00aa00aau;
  lo ^= t ^ (t << 7);
  t = (hi ^ (hi >> 7)) & 0x00aa00aau;
  hi ^= t ^ (t << 7);
  t = (lo ^ (lo >> 14)) & 0x0000ccccu;
  lo ^= t ^ (t << 14);
  t = (hi ^ (hi >> 14)) & 0x0000ccccu;
  hi ^= t ^ (t << 14);
  t = (lo ^ (hi << 4)) & 0xf0f0f0f0u;
  lo ^= t;
  hi ^= t >> 4;
}

// Bytes j of a, b, c, d -> word j.
__device__ __forceinline__ void transpose_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t* w) {
  const uint32_t ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);  // a0 b0 a1 b1
  const uint32_t ab2 = __byte_perm(a, b, 0x7362), cd2 = __byte_perm(c, d, 0x7362);
  w[0] = __byte_perm(ab, cd, 0x5410), w[1] = __byte_perm(ab, cd, 0x7632);
  w[2] = __byte_perm(ab2, cd2, 0x5410), w[3] = __byte_perm(ab2, cd2, 0x7632);
}

__global__ void __launch_bounds__(256, 4) mask_pack_kernel(const jvpfa_mask m, int n_h, int n_rows, int L, int n_qt, int n_words,
                                                        unsigned char* tile_live, int32_t* head_live,
                                                        unsigned long long* tile_live_t, int n_kt128, int n_words_t,
                                                        uint32_t* bits, uint32_t* bits_t) {
  __shared__ unsigned int s_tiles[2];                      // of the CTA's two 128-row tiles
  __shared__ uint32_t s_t[kPackKeys * 8 + kPackKeys / 8];  // [key][warp], one word of padding per 8 keys
  const int head = blockIdx.z, kg = blockIdx.x;            // kg: group of four key tiles
  const int b = head / n_h, h = head - b * n_h;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned char* base = reinterpret_cast<const unsigned char*>(m.ptr) + (long long)b * m.stride[0] + (long long)h * m.stride[1];
  const long long rs = m.stride[2], ks = m.stride[3];
  if (threadIdx.x < 2) s_tiles[threadIdx.x] = 0u;
  const int col = kg * kPackKeys + lane * 8;
  const int row0 = blockIdx.y * kPackRows + warp * 32;
  const bool vec = ks == 1 && (rs & 7) == 0 && (reinterpret_cast<uintptr_t>(base) & 7u) == 0 && col + 8 <= L;
  const unsigned char* p0 = base + (long long)row0 * rs + (long long)col * ks;
  uint32_t x[8];  // byte i of x[j]: row 4j + i, a bit per column
  if (vec) {
    // Sixteen rows in flight at a time, so that four CTAs fit an SM: one's loads run under another's arithmetic and stores
    // (B2 H12 L2048 from DRAM: 41 us with all 32 rows and two or three CTAs, 36 so).  Volatile loads: the compiler would move the
    // second half's before the first's arithmetic.
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint2 v[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        v[r] = make_uint2(0u, 0u);
        if (row0 + 16 * half + r < n_rows)
          asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v[r].x), "=r"(v[r].y) : "l"(p0 + (long long)(16 * half + r) * rs));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[4 * half + j] = 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) x[4 * half + j] |= (nonzero_bits(v[4 * j + i].x) | nonzero_bits(v[4 * j + i].y) << 4) << (8 * i);
      }
    }
  } else {
    // Rows that begin anywhere: three aligned words hold eight bytes of a row.  Where one of them would reach out of the mask, in its first
    // or last rows, the row's bytes are read one by one.  (All rows of such a lane were, one column after the other, and a launch takes as long
    // as its slowest warp.  From DRAM, us, before / so: 16 heads of L58 25 / 7, 77 of L66 11 / 7, 15 of L154 33 / 8, 43 of L130 11 / 8, 63 of
    // L338 21 / 9, 24 of L1330 31 / 21, of L2046 51 / 36, one of L4098 13 / 10.)
    // Where keys lie apart, or strides run backwards, byte by byte, in order of columns, so that all rows are in flight at once.
    const int n = min(8, L - col);  // <= 0: beyond the end
    const int rows = min(32, n_rows - row0);
    const unsigned char* first = reinterpret_cast<const unsigned char*>(m.ptr);
    const unsigned char* end = first + (long long)(gridDim.z / n_h - 1) * m.stride[0] + (long long)(n_h - 1) * m.stride[1] +
                               (long long)(n_rows - 1) * rs + (long long)(L - 1) * ks + 1;
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = 0u;
    if (ks == 1 && rs >= 0 && m.stride[0] >= 0 && m.stride[1] >= 0) {
      int r0 = 0, r1 = n > 0 ? max(rows, 0) : 0;  // rows [r0, r1): all of their words lie inside the mask
      const int r_end = r1;
      while (r1 > 0 && p0 + (long long)(r1 - 1) * rs + 12 > end) --r1;
      while (r0 < r1 && p0 + (long long)r0 * rs < first + 3) ++r0;
      const uint32_t cols = n > 0 ? (1u << n) - 1u : 0u;
      if (r0 < r1) {
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          uint32_t v[8][3], shift[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const unsigned char* p = p0 + (long long)(4 * j + r) * rs;
            shift[r] = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3u);
#pragma unroll
            for (int w = 0; w < 3; ++w) {
              v[r][w] = 0u;
              if (4 * j + r >= r0 && 4 * j + r < r1) v[r][w] = __ldg(reinterpret_cast<const uint32_t*>(p - shift[r]) + w);
            }
          }
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const uint32_t lo = __funnelshift_r(v[r][0], v[r][1], 8 * shift[r]), hi = __funnelshift_r(v[r][1], v[r][2], 8 * shift[r]);
            x[j + (r >> 2)] |= ((nonzero_bits(lo) | nonzero_bits(hi) << 4) & cols) << (8 * (r & 3));
          }
        }
      }
      for (int r = r0 > 0 ? 0 : r1; r < r_end; r = r + 1 == r0 ? r1 : r + 1) {
        uint32_t byte[8], set = 0u;
#pragma unroll
        for (int c = 0; c < 8; ++c) byte[c] = c < n ? __ldg(p0 + (long long)r * rs + c) : 0u;
#pragma unroll
        for (int c = 0; c < 8; ++c) set |= (byte[c] != 0u ? 1u : 0u) << c;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (r >> 2 == j) x[j] |= set << (8 * (r & 3));
      }
    } else {
      for (int c = 0; c < n; ++c) {
        uint32_t v[32];
#pragma unroll
        for (int r = 0; r < 32; ++r) {
          v[r] = 0u;
          if (r < rows) v[r] = __ldg(p0 + (long long)r * rs + (long long)c * ks);
        }
#pragma unroll
        for (int r = 0; r < 32; ++r) x[r >> 2] |= (v[r] != 0u ? 1u : 0u) << (8 * (r & 3) + c);
      }
    }
  }
  uint32_t any = 0u;
#pragma unroll
  for (int j = 0; j < 8; ++j) any |= x[j];
  const unsigned int vote = __ballot_sync(0xffffffffu, any != 0u);  // bit l: lane l saw a true entry
  if (bits != nullptr) {  // of four rows, lane l of four neighbours puts row l together: a 4 x 4 transpose of bytes across lanes
    const int w_rows = ((L + 63) / 64) * 2, word = kg * (kPackKeys / 32) + (lane >> 2);
    const uint32_t sel1 = lane & 1 ? 0x3715u : 0x6240u, sel2 = lane & 2 ? 0x3276u : 0x5410u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t y = __byte_perm(x[j], __shfl_xor_sync(0xffffffffu, x[j], 1), sel1);
      y = __byte_perm(y, __shfl_xor_sync(0xffffffffu, y, 2), sel2);
      const int row = row0 + 4 * j + (lane & 3);
      if (row < n_rows && word < w_rows) bits[((long long)head * n_rows + row) * w_rows + word] = y;
    }
  }
  __syncthreads();
  if (lane == 0 && vote != 0u) {
    unsigned int tiles = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (vote & (0xffu << (8 * k))) tiles |= 1u << k;
    atomicOr(&s_tiles[warp >> 2], tiles);
  }
  if (bits_t != nullptr) {
#pragma unroll
    for (int q = 0; q < 4; ++q) transpose8(x[2 * q], x[2 * q + 1]);  // byte c: column c (the second word: 4 + c) of eight rows
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t t[4];  // columns 4i .. 4i+3, a bit per row
      transpose_bytes(x[i], x[2 + i], x[4 + i], x[6 + i], t);
#pragma unroll
      for (int j = 0; j < 4; ++j) s_t[(lane * 8 + 4 * i + j) * 8 + warp + lane] = t[j];
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_tiles[threadIdx.x] != 0u && tile_live != nullptr) {
    const unsigned int tiles = s_tiles[threadIdx.x];
    const int qt = blockIdx.y * 2 + threadIdx.x;
    // tiles 4 kg .. 4 kg + 3 of the entry's words
    atomicOr(reinterpret_cast<unsigned int*>(tile_live) + ((long long)head * n_qt + qt) * n_words * 2 + (kg >> 3), tiles << (4 * (kg & 7)));
    if (head_live) {
      head_live[head] = 1;
      atomicAdd(head_live + gridDim.z, __popc(tiles));  // live tiles of the whole mask
    }
    if (tile_live_t) {  // the transposed summary: per 128-key tile, one bit per 128-query tile
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if ((tiles >> (2 * j)) & 3u)
          atomicOr(tile_live_t + ((long long)head * n_kt128 + 2 * kg + j) * n_words_t + (qt >> 6), 1ull << (qt & 63));
    }
  }
  if (bits_t != nullptr) {
    const int k = threadIdx.x, key = kg * kPackKeys + k;
    if (key >= L) return;
    const uint32_t* src = s_t + k * 8 + (k >> 3);
    if (n_rows == 1) {  // one row for every query: all bits of the key's only word alike
      bits_t[(long long)head * L + key] = (src[0] & 1u) ? ~0u : 0u;
      return;
    }
    const int w_cols = ((n_rows + 63) / 64) * 2, w0 = blockIdx.y * (kPackRows / 32);
    uint2* dst = reinterpret_cast<uint2*>(bits_t + ((long long)head * L + key) * w_cols + w0);
#pragma unroll
    for (int w = 0; w < 4; ++w)
      if (w0 + 2 * w < w_cols) dst[w] = make_uint2(src[2 * w], src[2 * w + 1]);
  }
}

// Eight elements (16 bytes stored) a lane at a time, kPadUnroll such pieces of a lane in flight: COLS of them along a row, by LANES lanes, the others
// on rows of the same head below it.  HBM bound: reads and writes two bytes an element.  Rows begin at any multiple of an element; PAIRS: two are one
// load, where all rows begin at a multiple of two (an even length).  The generic strided copy that it stands for looks each element's place up by
// itself: from DRAM on a B200, copy / this, us: B2 H3 L3698 (82 million elements) 188 / 59, B2 H11 L1450 110 / 37, B2 H12 L698 33 / 14.  (A warp for a row
// whatever its length left most pieces of short ones empty, and worked out each row's head: B1 H256 L98 16.4, copy 12.3, this 8.1; L178 24.6, 24.6,
// 12.3; B4 H16 L250 12.3, 16.4, 10.2; 800 calls of L 66 to 1400 with a bias, whole launches: 1.04 to 1.2 times as fast as with it in the mean, up to 1.8.)
constexpr int kPadUnroll = 4;
template <int LANES, int COLS, bool PAIRS>
__global__ void __launch_bounds__(256) pad_bias_kernel(const jvpfa_mask m, int n_h, int L, int width, uint32_t chunks, uint16_t* out) {
  constexpr int STEP = 32 / LANES, ROWS = STEP * (kPadUnroll / COLS);  // rows of a warp at a time, and in all
  const uint32_t head = blockIdx.x / chunks;
  const int b = (int)(head / (uint32_t)n_h), h = (int)(head - (uint32_t)b * (uint32_t)n_h);
  const int lane = threadIdx.x & 31, i0 = (int)(blockIdx.x - head * chunks) * 8 * ROWS + (int)(threadIdx.x >> 5) * ROWS + lane / LANES;
  const long long ks = m.stride[3];
  const uint16_t* src = reinterpret_cast<const uint16_t*>(m.ptr) + b * m.stride[0] + h * m.stride[1];
  uint16_t* dst = out + (size_t)head * L * width;
  for (int p0 = lane % LANES * 8; p0 < width; p0 += 8 * LANES * COLS) {
    uint32_t w[kPadUnroll][4];
#pragma unroll
    for (int u = 0; u < kPadUnroll; ++u) {
      const int i = i0 + u / COLS * STEP, j0 = p0 + 8 * LANES * (u % COLS), n = i < L ? L - j0 : 0;  // entries from j0 on
      const uint16_t* row = src + i * m.stride[2];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        w[u][e] = 0u;
        if (PAIRS && 2 * e + 1 < n) {
          w[u][e] = __ldg(reinterpret_cast<const uint32_t*>(row + j0 + 2 * e));
        } else {
          if (2 * e < n) w[u][e] = __ldg(row + (j0 + 2 * e) * ks);
          if (2 * e + 1 < n) w[u][e] |= (uint32_t)__ldg(row + (j0 + 2 * e + 1) * ks) << 16;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kPadUnroll; ++u) {
      const int i = i0 + u / COLS * STEP, j0 = p0 + 8 * LANES * (u % COLS);
      if (i < L && j0 < width) *reinterpret_cast<uint4*>(dst + (size_t)i * width + j0) = make_uint4(w[u][0], w[u][1], w[u][2], w[u][3]);
    }
  }
}

template <int LANES, int COLS>
int launch_pad(const jvpfa_pad_bias_args& a, bool pairs, cudaStream_t stream) {
  constexpr int ROWS = 8 * (32 / LANES) * (kPadUnroll / COLS);  // of a block
  const long long chunks = (a.L + ROWS - 1) / ROWS, blocks = (long long)a.n_b * a.n_h * chunks;
  if (blocks > 0x7fffffffLL) return JVPFA_ERR_TOO_LARGE;
  auto kern = pairs ? pad_bias_kernel<LANES, COLS, true> : pad_bias_kernel<LANES, COLS, false>;
  kern<<<(unsigned)blocks, 256, 0, stream>>>(a.mask, a.n_h, a.L, a.width, (uint32_t)chunks, static_cast<uint16_t*>(a.out));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "launch pad_bias");
    return JVPFA_ERR_CUDA;
  }
  return JVPFA_OK;
}

}  // namespace

// As many lanes to a row, and pieces along it, as it has.
int launch_pad_bias(const jvpfa_pad_bias_args& a, cudaStream_t stream) {
  bool pairs = a.mask.stride[3] == 1 && (reinterpret_cast<uintptr_t>(a.mask.ptr) & 3u) == 0;
  for (int d = 0; d < 3; ++d) pairs = pairs && (a.mask.stride[d] & 1) == 0;
  if (a.width <= 128) return launch_pad<16, 1>(a, pairs, stream);
  if (a.width <= 256) return launch_pad<32, 1>(a, pairs, stream);
  if (a.width <= 512) return launch_pad<32, 2>(a, pairs, stream);
  return launch_pad<32, 4>(a, pairs, stream);
}

int launch_mask_tiles(const jvpfa_mask_tiles_args& a, cudaStream_t stream) {
  const int n_kt = (a.L + 63) / 64;
  const int n_words = (n_kt + 63) / 64;
  const int n_qt = a.n_rows == 1 ? 1 : (a.L + 127) / 128;
  const dim3 grid((unsigned)((n_kt + 3) / 4), (unsigned)((a.n_rows + kPackRows - 1) / kPackRows), (unsigned)(a.n_b * a.n_h));
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
