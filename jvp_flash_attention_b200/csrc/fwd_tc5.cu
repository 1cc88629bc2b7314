// What the tcgen05 kernels share on the host side: the device status word of the bounded waits (with its host-visible
// mirror), the TMA tensor-map encoders, and the forward dispatch
//   D <= 64 -> fwd_tc5_pair64.cu  (two query tiles per CTA share every key stage)
//   D = 128 -> fwd_tc5_pipe128.cu (score products of the next key tile under the softmax of this one)
// Both follow the register-tiled kernel in fwd_generic.cu in what they compute (jvp_attention.py:125-336, 1011-1033).
#include <mutex>

#include "tc5_common.cuh"

namespace jvpfa {

// [0]: the status word.  [1]: kF32GaveUp.  [2], [3]: device address of its host-visible mirror (pinned, mapped host memory), written by
// a thread that gives up a wait, so that the host can see a failure without synchronising.
__device__ __align__(16) int g_tc5_status[4] = {0, 0, 0, 0};

namespace {
struct StatusSlot {
  int* dev = nullptr;            // device address of g_tc5_status on that device
  volatile int* mirror = nullptr;  // host address of the mirror (null if it could not be set up)
};
StatusSlot* status_slot() {
  static StatusSlot cache[64];
  static std::mutex setup;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  StatusSlot& sl = cache[dev];
  if (__atomic_load_n(&sl.dev, __ATOMIC_ACQUIRE)) return &sl;
  std::lock_guard<std::mutex> lock(setup);  // (calls are launched without the interpreter lock)
  if (!sl.dev) {
    int* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_tc5_status) != cudaSuccess) return nullptr;
    int* host = nullptr;
    int* host_dev = nullptr;
    if (cudaHostAlloc(reinterpret_cast<void**>(&host), sizeof(int), cudaHostAllocMapped) == cudaSuccess) {
      *host = 0;
      if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&host_dev), host, 0) == cudaSuccess &&
          cudaMemcpy(p + 2, &host_dev, sizeof(host_dev), cudaMemcpyHostToDevice) == cudaSuccess) {
        sl.mirror = host;
      } else {
        cudaFreeHost(host);
      }
    }
    (void)cudaGetLastError();  // a missing mirror only costs the early warning
    __atomic_store_n(&sl.dev, p, __ATOMIC_RELEASE);
  }
  return &sl;
}
}  // namespace

// Device address of the status word on the current device (other translation units receive it
// as a kernel argument).  Looked up once per device.
int* tc5_status_device_ptr() {
  StatusSlot* sl = status_slot();
  return sl ? sl->dev : nullptr;
}

// The mirror's value: non-zero once a kernel on the current device has given up a wait (no CUDA call, no
// synchronisation; it can lag behind the device by the kernels still in flight).
int tc5_status_peek() {
  StatusSlot* sl = status_slot();
  return (sl && sl->mirror) ? *sl->mirror : 0;
}

namespace tc5 {

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static const EncodeTiledFn fn = []() -> EncodeTiledFn {  // (once, and whoever comes meanwhile waits for it)
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
  }();
  return fn;
}

// The encoder is a driver call and wants a current context, which a thread that has made no runtime call yet does not have (its
// memory may come from an allocator's cache): it is given its device's then.
template <typename Encode>
static bool encode_in_context(Encode encode) {
  if (encode() == CUDA_SUCCESS) return true;
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && encode() == CUDA_SUCCESS;
}

bool encode_map4d(CUtensorMap* m, CUtensorMapDataType dt, const void* ptr, int D, int L, int H, int B, const int64_t* st,
                  int box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  const bool dense = st == nullptr || (st[0] == 0 && st[1] == 0 && st[2] == 0);
  const cuuint64_t sb = dense ? (cuuint64_t)H * L * D : (cuuint64_t)st[0];
  const cuuint64_t sh = dense ? (cuuint64_t)L * D : (cuuint64_t)st[1];
  const cuuint64_t sl = dense ? (cuuint64_t)D : (cuuint64_t)st[2];
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)L, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {sl * 2, sh * 2, sb * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_in_context([&]() {
    return fn(m, dt, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

// Row-major fp32 (B, H, L, D) tensor as a 4-D map with 32-column (128-byte) swizzled boxes: target of TMA reductions.
bool encode_map4d_f32(CUtensorMap* m, const void* ptr, int D, int L, int H, int B, int box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)L, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 4, (cuuint64_t)L * D * 4, (cuuint64_t)H * L * D * 4};
  cuuint32_t box[4] = {32, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_in_context([&]() {
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

bool encode_map_bias(CUtensorMap* m, CUtensorMapDataType dt, const jvpfa_mask& mask, int L, int H, int B, int box_rows) {
  const int64_t* ms = mask.stride;
  const int64_t st[3] = {ms[0] ? ms[0] : 8, ms[1] ? ms[1] : 8, ms[2] ? ms[2] : 8};  // (8: of one entry, not used)
  return encode_map4d(m, dt, mask.ptr, L, ms[2] ? L : 1, ms[1] ? H : 1, ms[0] ? B : 1, st, box_rows);
}

bool encode_map_parts(CUtensorMap* m, const void* ptr, int D, int L, int BH, int planes) {
  return encode_map4d(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, ptr, D, L, BH, planes, nullptr, 64);
}

}  // namespace tc5

// Head dimension 32 runs on the D = 64 kernels: the tensor maps end at column 32, so TMA fills the other half of every tile with zeros and clips what is stored, and the contractions over D stop
// half-way.  An MMA costs the same for 32 output columns as for 64, so little is wasted (B4 H8 L1000, bf16: forward with tangents
// 150 -> 46 us, backward through both outputs 325 -> 99 us in two launches, 58 in one, against the register-tiled kernels).  Up to one 64-row tile the
// register-tiled kernels stay: a 256-row pair of query tiles would be mostly padding.
bool tc5_head_dim(int D, int L) { return D == 64 || D == 128 || (D == 32 && L > 64); }

bool fwd_tc5_eligible(const jvpfa_fwd_args& a) {
  if (a.dtype != JVPFA_BF16 && a.dtype != JVPFA_FP16) return false;
  if (!tc5_head_dim(a.D, a.L)) return false;
  // The D <= 64 kernel takes the row maximum before scaling and therefore needs a positive softmax scale (any other
  // goes to the register-tiled kernels).
  if (a.D <= 64 && !(a.sm_scale > 0.f)) return false;
  const int k = a.mask.kind;
  if (k == JVPFA_MASK_NONE || k == JVPFA_MASK_CAUSAL || k == JVPFA_MASK_KVLEN) return true;
  return (k == JVPFA_MASK_BOOL && a.mask_bits != nullptr) || tc5_mask_layout(a.mask, a.dtype, a.L);
}

// Boolean masks and bias of the tensors' type: the kernels read 16-byte pieces of mask rows, the last piece of a row as
// well when only its head lies inside the row (what is beyond key L is then switched off by index).  That takes rows
// padded to whole pieces, which the native layer makes of a bias whose length does not fill them.
bool tc5_mask_layout(const jvpfa_mask& m, int dtype, int L) {
  if (m.kind == JVPFA_MASK_BIAS && m.bias_dtype != dtype) return false;
  const long long esz = m.kind == JVPFA_MASK_BOOL ? 1 : 2;
  if (m.stride[3] != 1 || (reinterpret_cast<uintptr_t>(m.ptr) & 15u) != 0) return false;
  for (int d = 0; d < 3; ++d)
    if (m.stride[d] < 0 || ((m.stride[d] * esz) & 15) != 0) return false;
  return (L & 15) == 0 || (m.stride[2] * esz >= ((L * esz + 15) & ~15ll));
}

// With the exact running maximum as its reference a row's largest probability is 1, which 16 bits hold without rounding;
// with a reference up to 2^8 below it (lazy rescaling) it is rounded like the others.  At a few hundred keys that is a part
// of the error that shows: O against 64 bits, B2 H4 D32, L512 fp16 with bias 2.56e-4 -> 2.90e-4, L1000 bf16 2.21e-3 ->
// 2.33e-3.  What the register-tiled kernels (exact) served before these kernels could, keeps their error: head dimension
// 32, and masks and bias that cannot be read in place as whole 16-byte pieces of rows (B4 H8 L1000 D32: forward with tangents
// 40 -> 46 us; B2 H12 L1330 D64 with bias 183 -> 191 us).
static bool exact_row_max(const jvpfa_fwd_args& a) {
  if (a.D == 32) return true;
  const bool by_element = a.mask.kind == JVPFA_MASK_BOOL || a.mask.kind == JVPFA_MASK_BIAS;
  return by_element && ((a.L & 15) != 0 || !tc5_mask_layout(a.mask, a.dtype, a.L));
}

int launch_fwd_tc5(const jvpfa_fwd_args& args, cudaStream_t s) {
  jvpfa_fwd_args a = args;
  if (exact_row_max(a)) a.flags |= tc5::kExactRowMax;
  if (a.D <= 64) return launch_fwd_tc5_pair64(a, s);
  return launch_fwd_tc5_pipe128(a, s);
}

int tc5_read_status(int* out, int clear) {
  StatusSlot* sl = status_slot();
  if (!sl) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  int v = 0;
  cudaError_t e = cudaMemcpy(&v, sl->dev, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "cudaMemcpy(status)");
    return JVPFA_ERR_CUDA;
  }
  if (clear && v != 0) {
    const int zero[2] = {0, 0};
    e = cudaMemcpy(sl->dev, zero, sizeof(zero), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      set_last_cuda_error(e, "cudaMemcpy(status)");
      return JVPFA_ERR_CUDA;
    }
    if (sl->mirror) *sl->mirror = 0;
  }
  *out = v;
  return JVPFA_OK;
}

// Puts `code` into the status word and its mirror from the host, as a kernel that gave up a wait would.
int tc5_inject_status(int code) {
  StatusSlot* sl = status_slot();
  if (!sl) {
    set_last_cuda_error(cudaErrorUnknown, "status word address");
    return JVPFA_ERR_CUDA;
  }
  cudaError_t e = cudaMemcpy(sl->dev, &code, sizeof(int), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    set_last_cuda_error(e, "cudaMemcpy(status)");
    return JVPFA_ERR_CUDA;
  }
  if (sl->mirror) *sl->mirror = code;
  return JVPFA_OK;
}

}  // namespace jvpfa
