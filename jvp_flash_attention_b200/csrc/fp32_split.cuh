// fp32 products on the 16-bit tensor-core path: tiles of fp16 pairs.
//
// A row of D floats is held as x = 2^-k (hi + lo), hi = fp16(2^k x), lo = fp16(2^k x - hi): 22 significant bits, as many
// as a pair of TF32 numbers has.  The exponent k is the row's own, chosen so that its largest entry lies in
// [2^14, 2^15): an entry keeps its 22 bits down to 2^-17 of that, and below it the error is at most 2^-40 of the largest.
// A product is lo*hi + hi*lo + hi*hi, each exact in the tensor core's fp32 accumulator.
//
// Why not TF32: mma.sync multiplies fp16 at twice the rate (1024 against 512 multiply-adds per clock and SM), a pair takes
// the space of the float it replaces, ldmatrix fetches whole fragments of it (transposed ones too), and the split is paid
// once per tile instead of once per warp that reads the tile.
//
// Where a row index is summed over (the keys in P V, the queries in P^T gO) the row's 2^-k goes into the other operand,
// whose rows are scaled again by their own largest entry: what a masked-out key or query holds then costs nobody
// precision, however large it is.
//
// Layout in shared memory: a row is D/8 pairs of 16-byte pieces, {8 hi, 8 lo} (the other way round in every second group
// of four pairs, which lets the threads that split a row reach all banks); piece p of row r lies at piece p ^ (r & 7) of
// the row, so that ldmatrix (eight rows, one piece of each) is free of bank conflicts.  The 32 bytes of a pair are those
// of the eight floats that become it, copied in by the thread that splits them in place.
#pragma once

#include "common.cuh"

namespace jvpfa {
namespace f32 {

// 2^k with which the largest magnitude m of a row lands in [2^14, 2^15), and 2^-k; both finite for every m.
__device__ __forceinline__ float row_scale(float m, float& inverse) {
  const int e = min(268 - (int)(__float_as_uint(m) >> 23), 253);
  inverse = __int_as_float((254 - e) << 23);
  return __int_as_float(e << 23);
}

__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x0, x1);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x0 - f.x, x1 - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

template <int D>
__device__ __forceinline__ uint32_t pair_offset(int row, int c) {  // of the piece with the hi parts; the other one: ^ 16
  return (uint32_t)row * (D * 4) + ((uint32_t)((2 * c) ^ ((c >> 2) & 1) ^ (row & 7)) << 4);
}

// Copies rows row0.. of a head (zeros at and beyond L) as floats; the same threads split them.
template <int ROWS, int D, int NT>
__device__ __forceinline__ void copy_tile(unsigned char* s, const float* head, int row0, int L, int tid, long long row_stride) {
  static_assert(ROWS * (D / 8) % 32 == 0, "whole warps");
#pragma unroll
  for (int idx = tid; idx < ROWS * (D / 8); idx += NT) {
    const int r = idx / (D / 8), c = idx % (D / 8), gr = row0 + r;
    const bool ok = gr < L;
    const float* src = head + (long long)(ok ? gr : 0) * row_stride + 8 * c;
    const uint32_t o = pair_offset<D>(r, c);
    cp_async16(s + o, src, ok ? 16 : 0);
    cp_async16(s + (o ^ 16u), src + 4, ok ? 16 : 0);
  }
}

// In place, after the thread's own copies have arrived; ROWS rows of one tile or of several that lie one after the other
// (each copied with copy_tile).  inv[row] = 2^-k.  The steps of one piece of work wait for one another (load, a maximum over
// the row's lanes, conversions), so up to four of them are taken at a time.
template <int ROWS, int TILE_ROWS, int D, int NT>
__device__ __forceinline__ void split_tiles(unsigned char* s, float* inv, int tid) {
  constexpr int kTile = TILE_ROWS * (D / 8);
  // the pairs that copy_tile gave this thread: tid, tid + NT, ... of every tile
  constexpr int kPer = (kTile + NT - 1) / NT, kMine = kPer * (ROWS / TILE_ROWS);
  constexpr int G = kMine % 4 == 0 ? 4 : kMine % 3 == 0 ? 3 : kMine % 2 == 0 ? 2 : 1;
  static_assert(kMine % G == 0 && ROWS % TILE_ROWS == 0, "whole batches");
#pragma unroll
  for (int w0 = 0; w0 < kMine; w0 += G) {
    float4 x[G], y[G];
    float m[G];
    uint32_t o[G];
    int row[G];
    bool on[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      const int w = w0 + i, in_tile = (w % kPer) * NT + tid;
      on[i] = kTile % NT == 0 || in_tile < kTile;  // the same for all lanes of a warp
      row[i] = (w / kPer) * TILE_ROWS + in_tile / (D / 8);
      o[i] = pair_offset<D>(row[i], in_tile % (D / 8));
      x[i] = y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on[i]) {
        x[i] = *reinterpret_cast<const float4*>(s + o[i]);
        y[i] = *reinterpret_cast<const float4*>(s + (o[i] ^ 16u));
      }
      m[i] = fmaxf(fmaxf(fmaxf(fabsf(x[i].x), fabsf(x[i].y)), fmaxf(fabsf(x[i].z), fabsf(x[i].w))),
                   fmaxf(fmaxf(fabsf(y[i].x), fabsf(y[i].y)), fmaxf(fabsf(y[i].z), fabsf(y[i].w))));
    }
#pragma unroll
    for (int d = D / 16; d > 0; d /= 2) {
#pragma unroll
      for (int i = 0; i < G; ++i) m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], d));
    }
#pragma unroll
    for (int i = 0; i < G; ++i) {
      float back;
      const float f = row_scale(m[i], back);
      uint4 hi, lo;
      split2(x[i].x * f, x[i].y * f, hi.x, lo.x);
      split2(x[i].z * f, x[i].w * f, hi.y, lo.y);
      split2(y[i].x * f, y[i].y * f, hi.z, lo.z);
      split2(y[i].z * f, y[i].w * f, hi.w, lo.w);
      if (on[i]) {
        *reinterpret_cast<uint4*>(s + o[i]) = hi;
        *reinterpret_cast<uint4*>(s + (o[i] ^ 16u)) = lo;
        if (tid % (D / 8) == 0) inv[row[i]] = back;
      }
    }
  }
}

struct PairA {
  uint32_t hi[4], lo[4];
};
struct PairB {
  uint32_t hi[2], lo[2];
};

template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  if constexpr (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// Rows r0..r0+15 (r0 a multiple of 8), columns k0..k0+15 of a tile at shared-memory address s.
template <int D>
__device__ __forceinline__ void load_a(PairA& f, uint32_t s, int r0, int k0, int lane) {
  const int row = r0 + (lane & 15);
  const uint32_t a = s + row * (D * 4) + ((uint32_t)((k0 / 4 + 2 * (lane >> 4)) ^ ((k0 / 32) & 1) ^ (lane & 7)) << 4);
  ldmatrix4<false>(a, f.hi[0], f.hi[1], f.hi[2], f.hi[3]);
  ldmatrix4<false>(a ^ 16u, f.lo[0], f.lo[1], f.lo[2], f.lo[3]);
}
// B operand of A * s^T: n = rows n0..n0+7, contraction over columns k0..k0+15.
template <int D>
__device__ __forceinline__ void load_b_nt(PairB& f, uint32_t s, int n0, int k0, int lane) {
  const uint32_t a = s + (n0 + (lane & 7)) * (D * 4) +
                     ((uint32_t)((k0 / 4 + 2 * ((lane >> 3) & 1) + (lane >> 4)) ^ ((k0 / 32) & 1) ^ (lane & 7)) << 4);
  ldmatrix4<false>(a, f.hi[0], f.hi[1], f.lo[0], f.lo[1]);
}
// B operand of A * s: contraction over rows k0..k0+15, n = columns n0..n0+7.
template <int D>
__device__ __forceinline__ void load_b_nn(PairB& f, uint32_t s, int k0, int n0, int lane) {
  const uint32_t a = s + (k0 + (lane & 15)) * (D * 4) + ((uint32_t)((n0 / 4 + (lane >> 4)) ^ ((n0 / 32) & 1) ^ (lane & 7)) << 4);
  ldmatrix4<true>(a, f.hi[0], f.hi[1], f.lo[0], f.lo[1]);
}

// One of the three instructions of a product: 0 = lo*hi, 1 = hi*lo, 2 = hi*hi.  Callers interleave the passes of several
// accumulators: an instruction returns some twenty cycles after it is issued.  FRESH: c starts from zero (as an operand of
// the instruction, not as four moves).
template <int PASS, bool FRESH = false>
__device__ __forceinline__ void mma_pass(float c[4], const PairA& a, const PairB& b) {
  const uint32_t* x = PASS == 0 ? a.lo : a.hi;
  const uint32_t* y = PASS == 1 ? b.lo : b.hi;
  if constexpr (FRESH)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(y[0]), "r"(y[1]), "f"(0.f));
  else
    mma_16816(static_cast<const __half*>(nullptr), c, x, y);
}

template <int N>
__device__ __forceinline__ void zero(float (*x)[4]) {
#pragma unroll
  for (int i = 0; i < N; ++i) x[i][0] = x[i][1] = x[i][2] = x[i][3] = 0.f;
}

// x[n-tile] = A0 B0^T, and where asked for y1 = A1 B0^T, y2 = A0 B1^T; 16 rows, 16 columns (two n-tiles), over D.
// AHEAD: the next step's operands are fetched ahead of this one's products (32 registers that two CTAs on an SM do not have,
// nor need: their warps cover for one another).
template <int D, bool HAS_Y1, bool HAS_Y2, bool AHEAD, int UNROLL = D / 16>
__device__ __forceinline__ void scores(float (*x)[4], float (*y1)[4], float (*y2)[4], uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1,
                                       int r0, int n0, int lane) {
  PairA fa0[2], fa1[2];
  PairB fb0[2][2], fb1[2][2];
  auto fetch = [&](int k0) {
    const int i = AHEAD ? (k0 / 16) & 1 : 0;
    load_a<D>(fa0[i], a0, r0, k0, lane);
    if constexpr (HAS_Y1) load_a<D>(fa1[i], a1, r0, k0, lane);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      load_b_nt<D>(fb0[i][n], b0, n0 + 8 * n, k0, lane);
      if constexpr (HAS_Y2) load_b_nt<D>(fb1[i][n], b1, n0 + 8 * n, k0, lane);
    }
  };
  if constexpr (AHEAD) fetch(0);
#pragma unroll UNROLL
  for (int k0 = 0; k0 < D; k0 += 16) {
    const int i = AHEAD ? (k0 / 16) & 1 : 0;
    if constexpr (AHEAD) {
      if (k0 + 16 < D) fetch(k0 + 16);
    } else {
      fetch(k0);
    }
    auto pass = [&](auto P, auto FRESH) {
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        mma_pass<P(), FRESH() != 0>(x[n], fa0[i], fb0[i][n]);
        if constexpr (HAS_Y1) mma_pass<P(), FRESH() != 0>(y1[n], fa1[i], fb0[i][n]);
        if constexpr (HAS_Y2) mma_pass<P(), FRESH() != 0>(y2[n], fa0[i], fb1[i][n]);
      }
    };
    if (k0 == 0)
      pass(IntC<0>{}, IntC<1>{});
    else
      pass(IntC<0>{}, IntC<0>{});
    pass(IntC<1>{}, IntC<0>{}), pass(IntC<2>{}, IntC<0>{});
  }
}

// A operand of a second product from an accumulator tile x (16 rows x 16 columns): column j times cs[j], then every row
// by the power of two that its largest entry asks for.  back[0 / 1]: its inverse for row g / g + 8.
__device__ __forceinline__ void a_from_acc(PairA& f, float back[2], const float (*x)[4], const float* cs, int lane) {
  const int t = lane & 3;
  const float2 c0 = *reinterpret_cast<const float2*>(cs + 2 * t), c1 = *reinterpret_cast<const float2*>(cs + 8 + 2 * t);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float v0 = x[0][2 * r] * c0.x, v1 = x[0][2 * r + 1] * c0.y, v2 = x[1][2 * r] * c1.x, v3 = x[1][2 * r + 1] * c1.y;
    const float m = quad_max(fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3))));
    const float k = row_scale(m, back[r]);
    split2(v0 * k, v1 * k, f.hi[r], f.lo[r]);
    split2(v2 * k, v3 * k, f.hi[2 + r], f.lo[2 + r]);
  }
}

// out[D/8][4] += A0 B0 (+ A1 B1), contraction over 16 rows of the tiles.  The tensor core adds into its accumulator with
// truncation, and hundreds of such adds into a long-lived one show up as a bias of 1e-5: every contraction step is formed
// in fresh registers and added rounded (which is also where the rows' scales are taken back).
template <int D, bool HAS_0, bool HAS_1>
__device__ __forceinline__ void outputs(float (*out)[4], const PairA& a0, const float* k0, const PairA& a1, const float* k1, uint32_t b0,
                                        uint32_t b1, int row0, int lane) {
  constexpr int G = 4;
#pragma unroll
  for (int d0 = 0; d0 < D / 8; d0 += G) {
    float x[G][4], y[G][4];
    PairB f0[G], f1[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if constexpr (HAS_0) load_b_nn<D>(f0[i], b0, row0, (d0 + i) * 8, lane);
      if constexpr (HAS_1) load_b_nn<D>(f1[i], b1, row0, (d0 + i) * 8, lane);
    }
    auto pass = [&](auto P) {
#pragma unroll
      for (int i = 0; i < G; ++i) {
        if constexpr (HAS_0) mma_pass<P(), P() == 0>(x[i], a0, f0[i]);
        if constexpr (HAS_1) mma_pass<P(), P() == 0>(y[i], a1, f1[i]);
      }
    };
    pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
#pragma unroll
    for (int i = 0; i < G; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (HAS_0) out[d0 + i][e] = fmaf(x[i][e], k0[e >> 1], out[d0 + i][e]);
        if constexpr (HAS_1) out[d0 + i][e] = fmaf(y[i][e], k1[e >> 1], out[d0 + i][e]);
      }
    }
  }
}

// The forward's pair of outputs in one sweep over V: o += A0 B0, t += A1 B0 (+ A2 B1)   (O += P V, tO += W V + P tV).
template <int D, bool HAS_2>
__device__ __forceinline__ void outputs_dual(float (*o)[4], float (*t)[4], const PairA& a0, const float* k0, const PairA& a1, const float* k1,
                                             const PairA& a2, const float* k2, uint32_t b0, uint32_t b1, int row0, int lane) {
  constexpr int G = 2;
#pragma unroll
  for (int d0 = 0; d0 < D / 8; d0 += G) {
    float x[G][4], y[G][4], z[G][4];
    PairB f0[G], f1[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      load_b_nn<D>(f0[i], b0, row0, (d0 + i) * 8, lane);
      if constexpr (HAS_2) load_b_nn<D>(f1[i], b1, row0, (d0 + i) * 8, lane);
    }
    auto pass = [&](auto P) {
#pragma unroll
      for (int i = 0; i < G; ++i) {
        mma_pass<P(), P() == 0>(x[i], a0, f0[i]);
        mma_pass<P(), P() == 0>(y[i], a1, f0[i]);
        if constexpr (HAS_2) mma_pass<P(), P() == 0>(z[i], a2, f1[i]);
      }
    };
    pass(IntC<0>{}), pass(IntC<1>{}), pass(IntC<2>{});
#pragma unroll
    for (int i = 0; i < G; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[d0 + i][e] = fmaf(x[i][e], k0[e >> 1], o[d0 + i][e]);
        t[d0 + i][e] = fmaf(y[i][e], k1[e >> 1], t[d0 + i][e]);
        if constexpr (HAS_2) t[d0 + i][e] = fmaf(z[i][e], k2[e >> 1], t[d0 + i][e]);
      }
    }
  }
}

// Rows row_lo + {0, 8} of a warp's accumulator strip, times f[0 / 1], to a row-major fp32 head.
template <int D>
__device__ __forceinline__ void store_strip(float* head, const float (*acc)[4], const float f[2], int row_lo, int L, int lane) {
  const int t = lane & 3;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = row_lo + 8 * r;
    if (row >= L) continue;
#pragma unroll
    for (int d = 0; d < D / 8; ++d)
      *reinterpret_cast<float2*>(head + (size_t)row * D + d * 8 + 2 * t) = make_float2(acc[d][2 * r] * f[r], acc[d][2 * r + 1] * f[r]);
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Rows x loop parts of a CTA.  A warp takes 16 rows and 16 rows of every loop tile, so a tile has 16 KG rows.  64 rows share
// every tile that is brought in, so they are the choice once they give each of the 148 SMs a CTA; below that shorter row
// tiles, whose warps share out the loop, put more SMs to work.  (D = 128 has no room for a loop tile of 128 rows.)
template <int D, typename F>
int dispatch_split(int B, int H, int L, F&& f) {
  const long long rows16 = (long long)((L + 15) / 16) * B * H;
  if (rows16 < 2 * 148) return f(IntC<1>{}, IntC<(D > 64 ? 4 : 8)>{});
  if (rows16 < 4 * 148) return f(IntC<2>{}, IntC<4>{});
  return f(IntC<4>{}, IntC<2>{});
}

}  // namespace f32
}  // namespace jvpfa
