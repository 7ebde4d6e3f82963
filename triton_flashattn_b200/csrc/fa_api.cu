// extern "C" entry points of libfa_sm100.so: argument validation, tensor-map
// encoding, the per-device status word and dispatch to the kernel launchers.
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "fa_host.cuh"

namespace fa {

// One status word per device that loads the library (file-scope device storage).
__device__ int g_fa_status[8];

std::atomic<uint64_t> g_kernel_launches{0};

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

constexpr int kMaxDevices = 64;
int* g_status_ptr[kMaxDevices];
volatile int32_t* g_mirror_host[kMaxDevices];  // pinned host copies of the status words
std::mutex g_status_mu;

struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  cudaError_t err = cudaSuccess;
  explicit DeviceGuard(int dev) {
    err = cudaGetDevice(&prev);
    if (err == cudaSuccess && prev != dev) {
      err = cudaSetDevice(dev);
      switched = (err == cudaSuccess);
    }
  }
  ~DeviceGuard() {
    if (switched) cudaSetDevice(prev);
  }
};

}  // namespace

int make_tmap_4d(CUtensorMap* out, const void* base, int elem_bytes, const uint64_t dims[4],
                 const uint64_t strides_bytes[3], const uint32_t box[4]) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return FA_ERR_CUDA;
  if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return FA_ERR_ALIGN;
  for (int i = 0; i < 3; ++i)
    if (strides_bytes[i] % 16 != 0 || strides_bytes[i] == 0) return FA_ERR_ALIGN;
  // Encoding is a pure function of these arguments, and a training loop presents the same
  // handful of (address, shape, stride) combinations step after step: a small per-thread
  // cache answers them without calling into the driver (about fifteen maps per step).
  struct Key {
    uint64_t v[12];
    bool operator==(const Key& o) const { return memcmp(v, o.v, sizeof(v)) == 0; }
  };
  struct Entry {
    Key key;
    CUtensorMap map;
    bool valid;
  };
  constexpr int kSlots = 256;
  thread_local Entry cache[kSlots] = {};
  Key key = {{reinterpret_cast<uint64_t>(base), (uint64_t)elem_bytes, dims[0], dims[1], dims[2], dims[3],
              strides_bytes[0], strides_bytes[1], strides_bytes[2],
              ((uint64_t)box[0] << 32) | box[1], ((uint64_t)box[2] << 32) | box[3], 0}};
  uint64_t hsh = 0x9E3779B97F4A7C15ull;
  for (int i = 0; i < 11; ++i) hsh = (hsh ^ key.v[i]) * 0xBF58476D1CE4E5B9ull + (hsh >> 29);
  Entry& e = cache[(hsh >> 20) % kSlots];
  if (e.valid && e.key == key) {
    memcpy(out, &e.map, sizeof(CUtensorMap));
    return FA_OK;
  }
  cuuint64_t gdim[4] = {dims[0], dims[1], dims[2], dims[3]};
  cuuint64_t gstr[3] = {strides_bytes[0], strides_bytes[1], strides_bytes[2]};
  cuuint32_t bx[4] = {box[0], box[1], box[2], box[3]};
  cuuint32_t es[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt =
      elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16
                      : (elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT32);
  const auto encode = [&] {
    return fn(out, dt, 4, const_cast<void*>(base), gdim, gstr, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // The driver wants a context, and a thread that has made no runtime call yet (the autograd engine's in a program's
    // first backward) has none bound.  (A layout that it refuses is another error, and no reason to bind one.)
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  }
  if (r != CUDA_SUCCESS) return FA_ERR_CUDA;
  e.key = key;
  memcpy(&e.map, out, sizeof(CUtensorMap));
  e.valid = true;
  return FA_OK;
}

int persistent_grid(int n_tiles) {
  static int sm_count[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = 0;
  if (dev >= 0 && dev < kMaxDevices) sms = sm_count[dev];
  if (sms <= 0) {
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
    if (dev >= 0 && dev < kMaxDevices) sm_count[dev] = sms;
  }
  if (const char* cap = getenv("FA_MAX_CTAS")) {
    const int c = atoi(cap);
    if (c > 0 && c < sms) sms = c;
  }
  return n_tiles < sms ? (n_tiles < 1 ? 1 : n_tiles) : sms;
}

int* device_status_ptr(int device) {
  if (device < 0 || device >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_status_mu);
  if (!g_status_ptr[device]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_fa_status) != cudaSuccess) return nullptr;
    g_status_ptr[device] = static_cast<int*>(p);
  }
  return g_status_ptr[device];
}

namespace {

// Whether elements of a bias, a mask or a bias gradient can be loaded and stored one by one at this address: the kernels that
// take any layout do that.
bool element_aligned(const void* ptr, int bias_kind) {
  const uintptr_t size = bias_kind == FA_BIAS_BOOL ? 1 : bias_kind == FA_BIAS_F32 ? 4 : 2;
  return reinterpret_cast<uintptr_t>(ptr) % size == 0;
}

int validate_common(const fa_params* p) {
  if (!p) return FA_ERR_NULL;
  if (p->struct_size != sizeof(fa_params)) return FA_ERR_ABI;
  if (p->B < 1 || p->H < 1 || p->M < 1 || p->N < 1) return FA_ERR_SHAPE;
  if (!(p->D == 16 || p->D == 32 || p->D == 64 || p->D == 128 || p->D == 256)) return FA_ERR_SHAPE;
  if (p->dtype != FA_F16 && p->dtype != FA_BF16) return FA_ERR_DTYPE;
  if (p->bias_kind < FA_BIAS_NONE || p->bias_kind > FA_BIAS_F32) return FA_ERR_DTYPE;
  if (!p->q || !p->k || !p->v || !p->o || !p->lse) return FA_ERR_NULL;
  if (p->bias_kind != FA_BIAS_NONE && !p->bias) return FA_ERR_NULL;
  if ((int64_t)p->B * p->H > 65535) return FA_ERR_TOO_LARGE;
  if (p->bias_kind != FA_BIAS_NONE && !element_aligned(p->bias, p->bias_kind)) return FA_ERR_ALIGN;
  return FA_OK;
}

// `workspace`: dS may go to scratch slabs, so the call needs no ds16 tensor
int validate_bwd(const fa_params* p, bool workspace = false) {
  int r = validate_common(p);
  if (r) return r;
  if (!p->d_o || !p->dq || !p->dk || !p->dv || !p->delta) return FA_ERR_NULL;
  if (p->write_dbias) {
    if (p->bias_kind != FA_BIAS_SAME && p->bias_kind != FA_BIAS_F32) return FA_ERR_DTYPE;
    if (!p->dbias) return FA_ERR_NULL;
    if (!element_aligned(p->dbias, p->bias_kind)) return FA_ERR_ALIGN;
  }
  if (workspace) return FA_OK;
  if (p->bias_kind == FA_BIAS_F32 && !p->ds16) return FA_ERR_NULL;
  // head dim 256: dQ is always the streamed product over the 16-bit dS
  if (p->D == 256 && !(p->write_dbias && p->bias_kind == FA_BIAS_SAME) && !p->ds16) return FA_ERR_NULL;
  return FA_OK;
}

// ---- backward through dS slabs ------------------------------------------------------------
// Whether dS already has a place of its own: the gradient of a 16-bit bias is dS.
bool ds_is_dbias(const fa_params& p) { return p.write_dbias && p.bias_kind == FA_BIAS_SAME; }

int64_t slab_pitch(const fa_params& p) { return ((int64_t)p.N + 7) / 8 * 8; }
uint64_t slab_bytes(const fa_params& p) { return (uint64_t)slab_pitch(p) * p.M * 2; }

// What a backward in parts of n problems costs in the dK/dV stage.
struct PartsCost {
  static constexpr int kTurn = 48;  // the unit: a 48th of a turn of one work unit per SM
  const fa_params& p;
  int total, tiles, sms, pair;
  explicit PartsCost(const fa_params& p)
      : p(p), total(p.B * p.H), tiles((p.N + 127) / 128), sms(persistent_grid(1 << 30)), pair(dkdv_pair_work(p)) {}
  // Time the persistent grids need for all problems, n at a time: full turns, or what the longest CTA does where a
  // causal launch goes longest first.  (A causal unit is a heavy and a light tile.)
  int64_t turns(int n) const {
    auto of = [&](int problems) -> int64_t {
      if (problems == 0) return 0;
      if (p.causal && p.D <= 128)
        if (const DkdvPlan plan = plan_dkdv(p, problems, sms, false); plan.longest_first)
          return (static_cast<int64_t>(kTurn) * plan.span + pair - 1) / pair;
      const int64_t k = (int64_t)problems * tiles;
      return kTurn * (((p.causal ? (k + 1) / 2 : k) + sms - 1) / sms);
    };
    return total / n * of(n) + of(total % n);
  }
  // Every part costs about a third of a turn more for its two launches and its drained tail.
  int64_t cost(int n) const { return turns(n) + kTurn / 3 * ((total + n - 1) / n); }
  // Problems per part, at most `most`: the number of least cost.  Among thousands of small problems one more
  // or less changes little, and a few hundred numbers are looked at (all of them took up to 0.1 ms a call).
  int best(int most) const {
    if (most >= total) return total;
    int n = most;
    int64_t least = cost(most);
    const int step = most / 512 + 1;
    for (int k = most - step; k > most / 2; k -= step)
      if (const int64_t c = cost(k); c < least) least = c, n = k;
    return n;
  }
};

// The scratch a backward works best with: room for the dS of all problems, or of as many as
// kSlabCap holds: 48 at a sequence length of 4096, 12 at 8192, 3 at 16384, none from 28 k on, where
// the scratch would grow with the square of the length.
constexpr uint64_t kSlabCap = 3ull << 29;

// Whether a backward in parts of n problems is faster than one with the recomputing dQ kernel.  Without a turn
// lost that kernel costs more than the streamed product by a share of the dK/dV time that depends on what it
// recomputes: three products instead of one at D = 128, little more than the traffic of dS at D = 64, and the
// bias or mask.  Backward alone, bf16, recomputing / in parts, us (problems per part; "no": the rule refuses it):
//   D 128: H8 S16384 causal 1790 / 1723 (3)          H8 S16384 3230 / 3250 (3)
//          H8 S20480 causal 2960 / 4040 (1, no)      H5 S27000 causal 3400 / 3740 (1, no)
//          H6 S16384 causal 1383 / 1289 (3)          H14 S8192 causal, mask 1117 / 790 (9; 12 in pairs 952)
//   D 64:  B16 H32 S2048 2820 / 2759 (192)           the same causal 1838 / 1601 (185)
//          B4 H32 S4096 2692 / 2708 (46, no)         B2 H16 S8192 causal 1466 / 1403 (8, no)
//          H16 S8192 1312 / 1442 (12, no)            the same causal 817 / 710 (8; 12 in pairs 743)
//          H32 S12288 causal 3052 / 3271 (3, no)     B2 H12 S8192 causal, mask 1388 / 1160 (9; 12 in pairs 1193)
bool parts_pay(const fa_params& p, const PartsCost& parts, int n) {
  if (n >= parts.total) return true;  // the same launches as without slabs
  const int64_t percent = (p.D > 64 ? 25 : 2) + (p.causal ? 10 : 0) + (p.bias_kind != FA_BIAS_NONE ? 20 : 0);
  return 100 * parts.cost(n) <= parts.turns(parts.total) * (100 + percent) + 100 * PartsCost::kTurn / 3;
}

uint64_t bwd_workspace_bytes(const fa_params& p) {
  const uint64_t one = slab_bytes(p), fit = kSlabCap / one;
  if (ds_is_dbias(p)) return 0;
  // backwards in one launch use none; with an fp32 bias some workspace is what stands for ds16 in the checks
  if (small_takes(p.M, p.N, p.D) || one_tile_takes(p)) return p.bias_kind == FA_BIAS_F32 ? one : 0;
  const PartsCost parts(p);
  const int total = parts.total;
  int n = fit < 1 ? 0 : parts.best(fit > (uint64_t)total ? total : (int)fit);
  if (p.D == 256 || p.bias_kind == FA_BIAS_F32) {
    // no other dQ kernel exists: as many more problems as lose no more than a seventh in turns that are not full
    // (H4 S20480 D256 causal in parts of one 4799 us a training pass, of all 3743)
    if (n < 1) n = 1;
    const int64_t full = parts.turns(total);
    while (n < total && 6 * parts.turns(n) > 7 * full) ++n;
    return one * (uint64_t)n;
  }
  return n >= 1 && parts_pay(p, parts, n) ? one * (uint64_t)n : 0;
}

int bwd_in_parts(const fa_params& p, void* ws, uint64_t bytes, cudaStream_t s, int* st) {
  const uint64_t fit = bytes / slab_bytes(p);
  const int total = p.B * p.H;
  const int n = PartsCost(p).best(fit > (uint64_t)total ? total : (int)fit);
  for (int bh0 = 0; bh0 < total; bh0 += n) {
    const DsSlab slab = {ws, slab_pitch(p), bh0, n < total - bh0 ? n : total - bh0};
    if (int e = launch_bwd_dkdv(p, s, st, &slab)) return e;
    if (int e = launch_bwd_dq(p, s, st, &slab)) return e;
  }
  return FA_OK;
}

// All stages of a backward without scratch.
int bwd_whole(const fa_params& p, cudaStream_t s, int* st) {
  if (small_takes(p.M, p.N, p.D)) {
    if (int e = check_tiled_bias(p, true)) return e;
    return launch_small(p, true, s, st);
  }
  if (one_tile_takes(p)) return launch_bwd_one_tile(p, s, st);
  if (int e = launch_bwd_pre(p, s, st)) return e;
  if (int e = launch_bwd_dkdv(p, s, st)) return e;
  return launch_bwd_dq(p, s, st);
}

// The row copies count the bytes of a row, and places up to 16 bytes behind its end, in 32 bits.
bool row_fits_copy(int N, int elem_bytes) { return static_cast<int64_t>(N) * elem_bytes <= INT32_MAX - 16; }

template <typename F>
int with_device(int device, F&& f) {
  DeviceGuard g(device);
  if (g.err != cudaSuccess) return FA_ERR_CUDA;
  int* status = device_status_ptr(device);
  if (!status) return FA_ERR_CUDA;
  return f(status);
}

}  // namespace
}  // namespace fa

using namespace fa;

extern "C" {

int fa_version(void) { return FA_ABI_VERSION; }

uint64_t fa_launch_count(void) { return g_kernel_launches.load(std::memory_order_relaxed); }

const char* fa_status_string(int code) {
  switch (code) {
    case FA_OK: return "ok";
    case FA_ERR_ABI: return "fa_params.struct_size does not match this library";
    case FA_ERR_NULL: return "a required pointer is null";
    case FA_ERR_SHAPE: return "bad shape (sizes must be >= 1, head dim in {16,32,64,128,256})";
    case FA_ERR_DTYPE: return "bad dtype or bias kind";
    case FA_ERR_ALIGN: return "pointer or stride is not a multiple of 16 bytes";
    case FA_ERR_CUDA: return "a CUDA call failed";
    case FA_ERR_DEVICE_WAIT: return "a kernel abandoned a bounded wait";
    case FA_ERR_UNSUPPORTED: return "not supported by this build";
    case FA_ERR_TOO_LARGE: return "size exceeds a limit of this entry point";
    default: return "unknown error code";
  }
}

int fa_fwd(const fa_params* p, void* stream) {
  int r = validate_common(p);
  if (r) return r;
  return with_device(p->device,
                     [&](int* st) { return launch_fwd(*p, static_cast<cudaStream_t>(stream), st); });
}

int fa_fwd_takes_any_bias(int M, int D) { return decode_takes(M, D) ? 1 : 0; }

int fa_small_takes(int M, int N, int D) { return small_takes(M, N, D) ? 1 : 0; }

int fa_small_fwd(const fa_params* p, void* stream) {
  int r = validate_common(p);
  if (r) return r;
  if (!small_takes(p->M, p->N, p->D)) return FA_ERR_UNSUPPORTED;
  return with_device(p->device, [&](int* st) { return launch_small(*p, false, static_cast<cudaStream_t>(stream), st); });
}

int fa_small_bwd(const fa_params* p, void* stream) {
  int r = validate_bwd(p, true);
  if (r) return r;
  if (!small_takes(p->M, p->N, p->D)) return FA_ERR_UNSUPPORTED;
  if (p->write_dbias) {  // every element has a place of its own
    const int extent[3] = {p->B, p->H, p->M};
    for (int i = 0; i < 3; ++i)
      if (extent[i] > 1 && p->dbias_stride[i] <= 0) return FA_ERR_ALIGN;
  }
  fa_params q = *p;
  q.ds16 = nullptr;  // not used here, whatever it says
  return with_device(p->device, [&](int* st) { return launch_small(q, true, static_cast<cudaStream_t>(stream), st); });
}

int fa_pad_rows(void* dst, const int64_t dst_stride[3], const void* src, const int64_t src_stride[3], int elem_bytes, int B, int H,
                int M, int N, int device, void* stream) {
  if (!dst || !src || !dst_stride || !src_stride) return FA_ERR_NULL;
  if (B < 1 || H < 1 || M < 1 || N < 1) return FA_ERR_SHAPE;
  if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4) return FA_ERR_DTYPE;
  if (!row_fits_copy(N, elem_bytes)) return FA_ERR_TOO_LARGE;
  return with_device(device, [&](int*) {
    return launch_pad_rows(dst, dst_stride, src, src_stride, elem_bytes, B, H, M, N, static_cast<cudaStream_t>(stream));
  });
}

int fa_pack_rows(void* dst, const void* src, int64_t pitch, int elem_bytes, int64_t rows, int N, int device, void* stream) {
  if (!dst || !src) return FA_ERR_NULL;
  if (rows < 1 || N < 1 || pitch < N) return FA_ERR_SHAPE;
  if (elem_bytes != 2 && elem_bytes != 4) return FA_ERR_DTYPE;
  if (!row_fits_copy(N, elem_bytes)) return FA_ERR_TOO_LARGE;
  if (reinterpret_cast<uintptr_t>(src) % 2 != 0) return FA_ERR_ALIGN;
  return with_device(device, [&](int*) {
    return launch_pack_rows(dst, src, pitch, elem_bytes, rows, N, static_cast<cudaStream_t>(stream));
  });
}

int fa_bwd_pre(const fa_params* p, void* stream) {
  int r = validate_bwd(p);
  if (r) return r;
  return with_device(p->device, [&](int* st) {
    return launch_bwd_pre(*p, static_cast<cudaStream_t>(stream), st);
  });
}

int fa_bwd_dkdv(const fa_params* p, void* stream) {
  int r = validate_bwd(p);
  if (r) return r;
  return with_device(p->device, [&](int* st) {
    return launch_bwd_dkdv(*p, static_cast<cudaStream_t>(stream), st);
  });
}

int fa_bwd_dq(const fa_params* p, void* stream) {
  int r = validate_bwd(p);
  if (r) return r;
  return with_device(p->device, [&](int* st) {
    return launch_bwd_dq(*p, static_cast<cudaStream_t>(stream), st);
  });
}

int fa_bwd(const fa_params* p, void* stream) {
  int r = validate_bwd(p);
  if (r) return r;
  return with_device(p->device, [&](int* st) { return bwd_whole(*p, static_cast<cudaStream_t>(stream), st); });
}

uint64_t fa_bwd_workspace_bytes(const fa_params* p) {
  if (validate_common(p)) return 0;
  uint64_t bytes = 0;
  with_device(p->device, [&](int*) {
    bytes = bwd_workspace_bytes(*p);
    return (int)FA_OK;
  });
  return bytes;
}

int fa_bwd_workspace(const fa_params* p, void* workspace, uint64_t bytes, void* stream) {
  const bool slabs = p && workspace && !validate_common(p) && !ds_is_dbias(*p) && bytes >= slab_bytes(*p);
  int r = validate_bwd(p, slabs);
  if (r) return r;
  if (!slabs) return fa_bwd(p, stream);
  if (reinterpret_cast<uintptr_t>(workspace) % 16 != 0) return FA_ERR_ALIGN;
  return with_device(p->device, [&](int* st) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (small_takes(p->M, p->N, p->D) || one_tile_takes(*p)) {
      fa_params q = *p;
      q.ds16 = nullptr;  // the workspace stands for it, whatever it says
      return bwd_whole(q, s, st);
    }
    if (int e = launch_bwd_pre(*p, s, st)) return e;
    return bwd_in_parts(*p, workspace, bytes, s, st);
  });
}

int fa_last_device_status(int device, int32_t out[8]) {
  if (!out) return FA_ERR_NULL;
  return with_device(device, [&](int* st) {
    if (cudaDeviceSynchronize() != cudaSuccess) return (int)FA_ERR_CUDA;
    if (cudaMemcpy(out, st, 8 * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
      return (int)FA_ERR_CUDA;
    return out[0] == 0 ? (int)FA_OK : (int)FA_ERR_DEVICE_WAIT;
  });
}

int fa_reset_device_status(int device) {
  return with_device(device, [&](int* st) {
    if (cudaDeviceSynchronize() != cudaSuccess) return (int)FA_ERR_CUDA;
    // words 6..7 (address of the host copy) stay
    if (cudaMemset(st, 0, 6 * sizeof(int)) != cudaSuccess) return (int)FA_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_status_mu);
    if (volatile int32_t* h = g_mirror_host[device])
      for (int i = 0; i < 6; ++i) h[i] = 0;
    return (int)FA_OK;
  });
}

int fa_set_status_mirror(int device, int32_t* host_words) {
  return with_device(device, [&](int* st) {
    unsigned long long dev_addr = 0;
    if (host_words) {
      void* d = nullptr;
      if (cudaHostGetDevicePointer(&d, host_words, 0) != cudaSuccess) return (int)FA_ERR_CUDA;
      dev_addr = reinterpret_cast<unsigned long long>(d);
      for (int i = 0; i < 8; ++i) host_words[i] = 0;
    }
    if (cudaDeviceSynchronize() != cudaSuccess) return (int)FA_ERR_CUDA;
    if (cudaMemcpy(st + 6, &dev_addr, sizeof(dev_addr), cudaMemcpyHostToDevice) != cudaSuccess)
      return (int)FA_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_status_mu);
    g_mirror_host[device] = host_words;
    return (int)FA_OK;
  });
}

int fa_selftest_wait_timeout(int device, uint32_t limit_us, void* stream) {
  if (limit_us < 1 || limit_us > 100000) return FA_ERR_SHAPE;
  return with_device(device, [&](int* st) {
    return launch_selftest_timeout(limit_us, static_cast<cudaStream_t>(stream), st);
  });
}

int fa_selftest_umma(int mode, int dtype, const void* a, const void* b, void* c, int device,
                     void* stream) {
  if (!a || !b || !c) return FA_ERR_NULL;
  if (mode < 0 || mode > 4) return FA_ERR_SHAPE;
  if (dtype != FA_F16 && dtype != FA_BF16) return FA_ERR_DTYPE;
  return with_device(device, [&](int* st) {
    return launch_selftest(mode, dtype, a, b, c, static_cast<cudaStream_t>(stream), st);
  });
}

}  // extern "C"
