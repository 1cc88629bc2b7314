// Blackwell (sm_100a) building blocks used by the tcgen05 kernels: mbarriers with bounded
// waits, TMA tile loads, TMEM allocation / load / store, UMMA shared-memory and instruction
// descriptors, and single-thread tcgen05.mma issue.
//
// Every wait in here is bounded by a cycle budget.  When a wait gives up it records a code in
// a CTA-wide abort flag and in the device-global status word; all later waits of the CTA return
// at once, the CTA drains, frees its TMEM and exits, and CTAs that start afterwards exit
// immediately.  The host reads the word through jvpfa_device_status().
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace jvpfa {
namespace tc5 {

constexpr long long kWaitBudgetCycles = 1ll << 31;  // about one second at B200 clocks

enum AbortCode : int {
  kAbortNone = 0,
  kAbortQFull = 1,
  kAbortKvFull = 2,
  kAbortKvEmpty = 3,
  kAbortSFull = 4,
  kAbortPFull = 5,
  kAbortOFull = 6,
  kAbortAux = 7,
  kAbortBwdOwn = 8,
  kAbortBwdLoopFull = 9,
  kAbortBwdLoopEmpty = 10,
  kAbortBwdSFull = 11,
  kAbortBwdPFull = 12,
  kAbortBwdDone = 13,
};

template <typename T>
struct Fmt;
template <>
struct Fmt<__nv_bfloat16> {
  static constexpr int kIdesc = 1;
  static constexpr CUtensorMapDataType kTma = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
};
template <>
struct Fmt<__half> {
  static constexpr int kIdesc = 0;
  static constexpr CUtensorMapDataType kTma = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two accumulator words as a packed pair of fp32 values, and the three-input maximum.
__device__ __forceinline__ float2 pf2(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Read-only global loads and 16-bit unpacking used for user masks and bias.
template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w);
template <>
__device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <>
__device__ __forceinline__ float2 unpack2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}

// One 16-bit element (in the low half of h) as float.
template <typename T>
__device__ __forceinline__ float unpack1(uint32_t h);
template <>
__device__ __forceinline__ float unpack1<__nv_bfloat16>(uint32_t h) {
  return __uint_as_float(h << 16);
}
template <>
__device__ __forceinline__ float unpack1<__half>(uint32_t h) {
  return __half2float(__ushort_as_half((unsigned short)h));
}

__device__ __forceinline__ uint4 ldg_nc_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

__device__ __forceinline__ uint32_t ldg_nc_u8(const void* p) {
  uint32_t r;
  asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(r) : "l"(p));
  return r;
}
__device__ __forceinline__ uint32_t ldg_nc_u16(const void* p) {
  uint16_t r;
  asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(r) : "l"(p));
  return r;
}

// In jvpfa_fwd_args.flags of the forward kernels, set by their launch: the running maximum is the reference of every tile.
constexpr int kExactRowMax = 1 << 30;

// Boolean masks.  A mask packed by jvpfa_mask_tiles is read as words; otherwise its bytes are turned into the same words.
__device__ __forceinline__ uint2 ldg_nc_v2(const void* p) {
  uint2 r;
  asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ uint32_t ldg_nc_u32(const void* p) {
  uint32_t r;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(r) : "l"(p));
  return r;
}
// index of (b, h) among the mask's own heads, and the words of one of its packed rows
__device__ __forceinline__ long long mask_head(const jvpfa_mask& m, int b, int h, int H) {
  return (m.stride[0] ? (long long)b * (m.stride[1] ? H : 1) : 0) + (m.stride[1] ? h : 0);
}
__device__ __forceinline__ const uint32_t* mask_bit_row(const void* bits, const jvpfa_mask& m, long long head, int i, int L) {
  const long long row = m.stride[2] ? head * L + i : head;
  return reinterpret_cast<const uint32_t*>(bits) + row * (((L + 63) >> 6) * 2);
}
// ... and of one of its packed columns (a single word that stands for every query when the mask has one row)
__device__ __forceinline__ const uint32_t* mask_bit_col(const void* bits_t, const jvpfa_mask& m, long long head, int j, int L) {
  return reinterpret_cast<const uint32_t*>(bits_t) + (head * L + j) * (m.stride[2] ? ((L + 63) >> 6) * 2 : 1);
}
__device__ __forceinline__ uint32_t bits_of_bytes(uint32_t w) {  // bytes -> four bits
  return (((__vcmpne4(w, 0u) & 0x01010101u) * 0x01020408u) >> 24) & 0xfu;
}
// 16 mask bytes at p (a 16-byte piece that starts at key j of its row; 0 beyond the row) as 16 bits
__device__ __forceinline__ uint32_t mask_piece_bits(const unsigned char* p, int j, int L) {
  if (j >= L) return 0u;
  const uint4 r = ldg_nc_v4(p);
  return bits_of_bytes(r.x) | bits_of_bytes(r.y) << 4 | bits_of_bytes(r.z) << 8 | bits_of_bytes(r.w) << 12;
}
// the first n of 32 columns (n may be negative or beyond 32)
__device__ __forceinline__ uint32_t first_columns(int n) { return n >= 32 ? ~0u : n <= 0 ? 0u : (1u << n) - 1u; }

// Host: (D, L, H, B) view of a 16-bit tensor whose batch / head / row strides (in elements) are given
// (all zero: (B,H,L,D) row-major); box = 64 columns x box_rows rows (a D = 128 tile is two loads), 128-byte swizzle,
// out-of-range rows and columns read as zero.  Defined in fwd_tc5.cu.
bool encode_map4d(CUtensorMap* m, CUtensorMapDataType dt, const void* ptr, int D, int L, int H, int B, const int64_t* stride_bhl,
                  int box_rows);
// (keys, rows, heads, entries) view of a 16-bit bias whose rows are whole 16-byte pieces (tc5_mask_layout), box = 64 keys x box_rows rows;
// a dimension that broadcasts (stride 0) has one entry.
bool encode_map_bias(CUtensorMap* m, CUtensorMapDataType dt, const jvpfa_mask& mask, int L, int H, int B, int box_rows);
// Row-major fp32 (B, H, L, D) tensor, 32-column boxes with 128-byte swizzle (target of TMA reductions).
bool encode_map4d_f32(CUtensorMap* m, const void* ptr, int D, int L, int H, int B, int box_rows);

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void lds_v4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}

// ---- mbarrier ------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// ... when `v`, the word that a warp's last load from shared memory returns, is there (they return in their order).  An arrival does not wait for loads from shared memory in flight, and may
// overtake them: one that stood right behind a tile's last load (16 softmax warps, the smem port busy with the first tiles of a CTA) let
// the next tile be copied over what those loads had yet to read, once in about fifty launches.  The barrier's address is formed with v, of which
// `none` keeps no bit: a value that is zero in every launch and that no compiler knows (opaque_zero), so that nothing can take the arrival for one
// that does not depend on v.
__device__ __forceinline__ void mbar_arrive_behind(uint64_t* bar, uint32_t v, uint32_t none) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar) + (v & none)) : "memory");
}
// The sign of a launch's struct_size, which the host has compared with the size itself.
template <typename Args>
__device__ __forceinline__ uint32_t opaque_zero(const Args& a) {
  return (uint32_t)(a.struct_size >> 31);
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

struct AbortState {
  volatile int* cta_flag;  // shared memory
  int* global_status;      // device global
};

// What a wait that gives up leaves for everybody.  First failure wins; the code also goes to the host-visible mirror whose device address sits beside the status word
// (two ints further, 8-byte aligned), so that the host learns of it without synchronising.
__device__ __forceinline__ void publish_abort(int* global_status, int code) {
  if (atomicCAS(global_status, 0, code) == 0) {
    int* mirror = *reinterpret_cast<int* const*>(global_status + 2);
    if (mirror) {
      *reinterpret_cast<volatile int*>(mirror) = code;
      __threadfence_system();
    }
  }
}
__device__ __forceinline__ bool mbar_try_wait_u32(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// One look, without waiting.  (`quiet`: loads and stores may be moved across it; for barriers that guard nothing but what volatile
// instructions behind it touch.)
__device__ __forceinline__ uint32_t mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok;
}
__device__ __forceinline__ uint32_t mbar_test_quiet(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity));
  return ok;
}
// Bounded wait.  Returns false (and latches the abort state) when the budget runs out or when
// another thread of the CTA has already given up.  A measured mbarrier hand-off between two warps
// costs ~200 cycles.  Measured on the forward kernels (two CTAs per SM, many warps waiting at once):
// a poll loop that reads the clock right after the first failed attempt is ~5 % faster overall
// than one that polls 128 times first, which takes issue slots from the warps that compute.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const AbortState& ab, int code) {
  const uint32_t addr = smem_u32(bar);
  if (mbar_try_wait_u32(addr, parity)) return true;
  const long long t0 = clock64();
  int polls = 0;
  while (true) {
    if (mbar_try_wait_u32(addr, parity)) return true;
    if ((++polls & 63) == 0) {
      if (*ab.cta_flag != 0) return false;
      if (clock64() - t0 > kWaitBudgetCycles) {
        *ab.cta_flag = code;
        publish_abort(ab.global_status, code);
        return false;
      }
    }
  }
}
// For roles far from the critical path (a producer several stages ahead): sleeps between attempts, because every
// attempt is an access on the shared-memory port that the MMA operands come through.
template <int NS = 128>
__device__ __forceinline__ bool mbar_wait_backoff(uint64_t* bar, uint32_t parity, const AbortState& ab, int code) {
  const uint32_t addr = smem_u32(bar);
  if (mbar_try_wait_u32(addr, parity)) return true;
  const long long t0 = clock64();
  int polls = 0;
  while (true) {
    __nanosleep(NS);
    if (mbar_try_wait_u32(addr, parity)) return true;
    if ((++polls & 63) == 0) {
      if (*ab.cta_flag != 0) return false;
      if (clock64() - t0 > kWaitBudgetCycles) {
        *ab.cta_flag = code;
        publish_abort(ab.global_status, code);
        return false;
      }
    }
  }
}
// The wait of an issuing warp, by all of its lanes with one outcome for them (a lane that gave up takes the others along: what
// follows needs all of them).  A warp that stays converged keeps descriptors and loop counters in uniform registers, where
// tcgen05.mma takes its operands from, and only the instructions themselves are one lane's (`elect_one`).  Issued from a branch of
// lane 0 every operand is moved there first: measured on a B200, cycles per M = 128 instruction with such a branch / a converged
// warp: N = 64 with A in TMEM 45-54 / 32, both operands in shared memory 48-57 / 48 (what the port delivers), N = 32 45 / 40,
// N = 128 64 / 64.
__device__ __forceinline__ bool mbar_wait_warp_u32(uint32_t addr, uint32_t parity, const AbortState& ab, int code) {
  bool ok = true;
  if (!mbar_try_wait_u32(addr, parity)) {
    const long long t0 = clock64();
    int polls = 0;
    while (!mbar_try_wait_u32(addr, parity)) {
      if ((++polls & 63) == 0) {
        if (*ab.cta_flag != 0) {
          ok = false;
          break;
        }
        if (clock64() - t0 > kWaitBudgetCycles) {
          *ab.cta_flag = code;
          publish_abort(ab.global_status, code);
          ok = false;
          break;
        }
      }
    }
  }
  return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, const AbortState& ab, int code) {
  return mbar_wait_warp_u32(smem_u32(bar), parity, ab, code);
}
// One lane of the converged warp, always the same.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// ---- Key padding: the batch entries, longest first ----------------------------------------
// Persistent kernels deal their items in one order to all CTAs; with the entries' lengths mixed some CTAs got the long ones twice
// (B8 H12 L1024, lengths in [L/2, L], 148 CTAs: 39-48 key tiles in the forward against 32-40 for the longest first, mean 28-34;
// in the backward 6 key tiles of 128 against 5).  Up to this many entries, and where a CTA has more than one item.
constexpr int kMaxSortedBatch = 64;
// By all threads of the CTA, before they meet: order[r] = the r-th longest entry.
__device__ __forceinline__ void sort_batch(const jvpfa_mask& m, int B, unsigned char* order) {
  if ((int)threadIdx.x < B) {
    const int mine = m.kv_len[threadIdx.x];
    int r = 0;
    for (int x = 0; x < B; ++x) {
      const int n = m.kv_len[x];
      r += n > mine || (n == mine && x < (int)threadIdx.x);
    }
    order[r] = (unsigned char)threadIdx.x;
  }
}

// ---- Items shared out among CTAs --------------------------------------------------------------
// Persistent kernels whose items (each with a loop of n steps) would leave a round of CTAs half empty share their steps out: the items
// in a line, by head and by place in the head, cut into as many equal pieces as there are CTAs.  An item's beginning counts as `open`
// steps.  Item r of a head of batch entry b stands for first(b) + slope * r steps (it may have fewer), tiles(b) of the per_head items
// of a head stand in the line.  Where all items are alike, `whole` rounds of items are dealt whole and only the rest, from item whole * G on, is the line: fewer cuts.
constexpr int kMinPiece = 2;  // a cut leaves at least so many steps on either side
// By one whole warp: where CTA c of G begins, {head * per_head + r, step}.  steps(b, r): how many item r has.  The line's length times
// G fits 32 bits (cut_fits).
template <typename Tiles, typename First, typename Steps>
__device__ __forceinline__ int2 cut_begin(bool by_entry, int B, int H, int per_head, int slope, int open, int whole, int c, int G, Tiles tiles,
                                          First first, Steps steps) {
  const int lane = threadIdx.x & 31;
  if (c <= 0) return make_int2(whole * G, 0);
  if (c >= G) return make_int2(B * H * per_head, 0);
  if (!by_entry && slope == 0) {
    const int n = first(0), item = n + open;
    const int pos = (int)((unsigned)((B * H * per_head - whole * G) * item) * (unsigned)c / (unsigned)G);
    int w = pos / item, s = pos - w * item - open;
    if (s < kMinPiece) s = 0;
    if (s > n - kMinPiece) s = 0, ++w;
    return make_int2(whole * G + w, s);
  }
  auto upto = [&](int b, int r) { return r * (first(b) + open) + slope * (r * (r - 1) / 2); };
  int b = 0, pos;
  if (!by_entry) {  // all heads alike
    const int head = upto(0, tiles(0));
    pos = (int)((unsigned)(B * H * head) * (unsigned)c / (unsigned)G);
    b = pos / head / H;
    pos -= b * H * head;
  } else {
    auto batch = [&](int x) { return x < B ? H * upto(x, tiles(x)) : 0; };
    int total = 0;
    for (int x = lane; x < B; x += 32) total += batch(x);
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    pos = (int)((unsigned)total * (unsigned)c / (unsigned)G);
    b = B;
    for (int x0 = 0; x0 < B; x0 += 32) {  // the entry that holds this place of the line
      const int mine = batch(x0 + lane);
      int upto_me = mine;
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, upto_me, d);
        if (lane >= d) upto_me += o;
      }
      const unsigned beyond = __ballot_sync(0xffffffffu, upto_me > pos);
      if (beyond) {
        const int src = __ffs(beyond) - 1;
        b = x0 + src;
        pos -= __shfl_sync(0xffffffffu, upto_me - mine, src);
        break;
      }
      pos -= __shfl_sync(0xffffffffu, upto_me, 31);
    }
    if (b == B) return make_int2(B * H * per_head, 0);  // (an empty line)
  }
  const int T = tiles(b), head = upto(b, T);
  const int bh = b * H + pos / head;
  pos %= head;
  int lo = 0, hi = T - 1;  // the last item that begins at or before pos
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (upto(b, mid) <= pos) lo = mid; else hi = mid - 1;
  }
  int r = lo, s = pos - upto(b, r) - open;
  if (s < kMinPiece) s = 0;
  if (s > steps(b, r) - kMinPiece) s = 0, ++r;
  return make_int2(bh * per_head + r, s);
}
inline bool cut_fits(long long line, long long ctas) { return line * ctas < 1ll << 32 && line < 1ll << 31; }
// Items dealt whole in serpentine order to G CTAs: the load of the CTA that has most, of `looks` + 1 of them.  load(w): of item w.
template <typename Load>
long long most_loaded(long long items, long long G, int looks, Load load) {
  long long most = 0;
  for (int at = 0; at <= looks; ++at) {
    const long long c = (G - 1) * at / looks;
    long long sum = 0;
    for (long long k = 0; k * G < items; ++k) {
      const long long w = k * G + ((k & 1) ? G - 1 - c : c);
      if (w < items) sum += load(w);
    }
    most = sum > most ? sum : most;
  }
  return most;
}
// The lengths of a key padding on the host, for the rules: tiles of `tile` keys of the batch entry that whole items meet r-th (where the
// kernel sorts them by length, `sorted`, the r-th longest).
struct HostLengths {
  const int32_t* len;
  int L;
  bool sorted;
  unsigned char order[kMaxSortedBatch];
  HostLengths(const int32_t* l, int B, int L_, bool s) : len(l), L(L_), sorted(s) {
    for (int b = 0; s && b < B; ++b) {
      int r = b;
      for (; r > 0 && len[order[r - 1]] < len[b]; --r) order[r] = order[r - 1];
      order[r] = (unsigned char)b;
    }
  }
  long long tiles(long long r, int tile) const {
    const int n = len[sorted ? order[r] : r];
    return ((n < 0 ? 0 : n > L ? L : n) + tile - 1) / tile;
  }
};
// CTA c's place in the workspace for its share of item w, which is not its as a whole: 2 c where it takes the item over, else 2 c + 1;
// -1 where the whole item is its.  at: {item, step} where this CTA and the next begin.
__device__ __forceinline__ int cut_place(const int* at, int w, int c) {
  const bool before = w == at[0] && at[1] > 0;
  return before || w == at[2] ? 2 * c + (before ? 0 : 1) : -1;
}
// Calls add(place) for the shares, in their order, of the item that is cut first where CTA j begins; false, and no call, if no item is.
// begin: where each of the CTAs begins; item: the item.
template <typename Add>
__device__ __forceinline__ bool cut_shares(const int2* begin, int ctas, int j, int* item, Add add) {
  const int2 at = begin[j], before = begin[j - 1];
  if (at.y == 0 || (before.x == at.x && before.y > 0)) return false;
  *item = at.x;
  add(2 * (j - 1) + 1);  // the share that begins the item is its CTA's last
  int2 cur = at;
  for (int m = j; m < ctas; ++m) {
    const int2 next = m + 1 < ctas ? begin[m + 1] : make_int2(-1, 0);
    if (next.x != cur.x || next.y != cur.y) add(2 * m);  // (else CTA m has nothing to do)
    if (next.x != at.x || next.y == 0) break;
    cur = next;
  }
  return true;
}

// ---- TMA -----------------------------------------------------------------------------------
// Into L2 alone.
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y,
                                            int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- TMEM ----------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_commit_u32(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 32 lanes x 32 columns: thread i of the warp receives columns [col, col+32) of TMEM lane
// (warp % 4) * 32 + i.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
      "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
      "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ---- UMMA descriptors ----------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (sm_100).  Addresses and byte
// offsets are stored without their 4 low bits.
//   K-major operand  (rows of 64 16-bit elements = 128 B): 8-row groups are sbo bytes apart.
//   MN-major operand (same tile used transposed): 64-element chunks along MN are lbo bytes
//   apart, groups of 8 along K are sbo bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16, fp32 accumulation.  fmt: 0 = f16, 1 = bf16.
__host__ __device__ constexpr uint32_t make_idesc(int fmt, int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)a_mn_major << 15) |
         ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}


// The same two instructions with the shared-memory descriptors given as (low, high) words.  For the
// 128-byte-swizzled tiles used here (leading offset 16 B, 8-row groups 1024 B apart) the high word
// is the constant kDescHi and the low word is kDescLo | (byte address >> 4): stepping through a
// tile is an integer add on the low word.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
constexpr uint32_t kDescLo = (16u >> 4) << 16;
template <bool ACC>
__device__ __forceinline__ void umma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}
template <bool ACC>
__device__ __forceinline__ void umma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(kDescHi), "r"(idesc), "n"(ACC ? 1 : 0)
      : "memory");
}
// accumulate flag known only at run time
__device__ __forceinline__ void umma_ss_lo_dyn(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_ts_lo_dyn(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Outputs of a launch that ran after a bounded wait gave up (or of the launch that gave up) are undefined.  To make
// that visible without a synchronisation, such a CTA stamps NaN into the statistics / leading elements of the rows
// it owns: every later reduction over the outputs, and every backward that reads lse, then carries NaN.
__device__ __forceinline__ float poison_f32() { return __uint_as_float(0x7fc00000u); }
template <typename T>
__device__ __forceinline__ void poison_row(void* base, size_t row, int D) {  // first 16 bytes of a (.., D) row
  uint4* p = reinterpret_cast<uint4*>(reinterpret_cast<T*>(base) + row * D);
  *p = sizeof(T) == 2 ? make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu)
                      : make_uint4(0x7fc00000u, 0x7fc00000u, 0x7fc00000u, 0x7fc00000u);
}


}  // namespace tc5
}  // namespace jvpfa
