// Host-side helpers shared by the translation units of libfa_sm100.so: tensor-map
// encoding without linking libcuda, the per-device status word, and the launcher
// prototypes that fa_api.cu dispatches to.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/fa_sm100.h"

namespace fa {

// ---- tensor maps -----------------------------------------------------------
// 4-D tiled map over 16-bit (or 8-bit) elements with the 128-byte swizzle.
//   dims[0] is the innermost (unit stride) extent; strides_bytes[i] is the byte
//   stride of dims[i+1].  box[] is the tile copied per request.
// Returns FA_OK, FA_ERR_ALIGN (address/stride rule broken) or FA_ERR_CUDA.
int make_tmap_4d(CUtensorMap* out, const void* base, int elem_bytes, const uint64_t dims[4],
                 const uint64_t strides_bytes[3], const uint32_t box[4]);

// ---- status word -----------------------------------------------------------
// Device address of the int[8] status word of the current device (file-scope
// __device__ storage inside the library; nothing is allocated).
int* device_status_ptr(int device);

// ---- launchers (defined next to their kernels) -----------------------------
// A part of the (batch, head) problems, numbered b * H + h, with a 16-bit (M, pitch) slab of
// scratch for the dS of each: the dK/dV stage leaves dS there and the dQ stage streams it.
struct DsSlab {
  void* base;     // slab of problem bh0
  int64_t pitch;  // row pitch in elements, a multiple of 8
  int bh0, n_bh;
};

int launch_fwd(const fa_params& p, cudaStream_t stream, int* status);
// Forward for a few query rows: whether it takes the problem, and its launch.  It reads the bias
// element by element, so that needs no alignment there.
bool decode_takes(int M, int D);
int launch_decode(const fa_params& p, cudaStream_t stream, int* status);
// Short sequences: whether the kernels of fa_small.cu take the problem, and their launch.  They read the bias and write its
// gradient at any address, with any strides but the innermost; `check_tiled_bias` has what the tile kernels ask of them.
bool small_takes(int M, int N, int D);
int launch_small(const fa_params& p, bool bwd, cudaStream_t stream, int* status);
int check_tiled_bias(const fa_params& p, bool bwd);
// Row copies (fa_copy.cu); strides and pitch in elements of `eb` bytes.
int launch_pad_rows(void* dst, const int64_t dst_stride[3], const void* src, const int64_t src_stride[3], int eb, int B, int H, int M,
                    int N, cudaStream_t stream);
int launch_pack_rows(void* dst, const void* src, int64_t pitch, int eb, int64_t rows, int N, cudaStream_t stream);
int launch_bwd_pre(const fa_params& p, cudaStream_t stream, int* status);
// How a causal dK/dV launch of head dims up to 128 over `n_bh` problems walks its tiles (see plan_dkdv), and how long its
// longest CTA works then, in quarters of a step; 0 where that was not looked at (pairs, many tiles a CTA).
struct DkdvPlan {
  bool longest_first;
  int span;
};
DkdvPlan plan_dkdv(const fa_params& p, int n_bh, int sms, bool writes_zeros);
// Work of a pair of a heavy and a light tile in the same unit.
int dkdv_pair_work(const fa_params& p);
// Without a slab: all problems, dS going where the parameters say (dbias, ds16 or nowhere).
int launch_bwd_dkdv(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab = nullptr);
// The whole backward in one launch where one tile holds all keys: whether it takes the problem, and its launch.
bool one_tile_takes(const fa_params& p);
int launch_bwd_one_tile(const fa_params& p, cudaStream_t stream, int* status);
int launch_bwd_dq(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab = nullptr);
// Head dimension 256: its own dV kernel, which always leaves the 16-bit dS in global
// memory (in dbias for a 16-bit bias that wants its gradient, else in the ds16 scratch;
// d256_ds_tensor names that tensor), and dK and dQ as products that stream it.
int launch_bwd_dkdv_d256(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab);
int launch_bwd_dk_from_ds(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab);
const void* d256_ds_tensor(const fa_params& p, const int64_t** stride);
int launch_selftest(int mode, int dtype, const void* a, const void* b, void* c, cudaStream_t stream,
                    int* status);
int launch_selftest_timeout(uint32_t limit_us, cudaStream_t stream, int* status);

// Grid of a persistent kernel: one CTA per SM of the current device, never more than
// there are work units.  The environment variable FA_MAX_CTAS (a positive integer, read at
// every launch) lowers the cap; tests use it to make small problems walk many tiles
// per CTA.
int persistent_grid(int n_tiles);

// What the longest CTA of a causal launch has to do in the two orders in which persistent CTAs take its n units: n_bh
// heads of `levels` units each, work(level) falling from level 0 on.
//   pairs: the units of a head are ordered heavy, light, next heavy, next light, ..., and CTA c takes two neighbours in a
//     turn, pair c, c + G, ...
//   longest first: the units are numbered by level, heads inside it, and the CTAs take them in rows, every second row from
//     the other end.
struct CausalSpans {
  int pairs, longest_first;
};
template <typename Work>
inline CausalSpans causal_spans(int n, int n_bh, int levels, int sms, Work work) {
  CausalSpans span = {0, 0};
  const auto more = [](int& most, int load) { most = load > most ? load : most; };
  // Pairs: the work of a CTA's pairs repeats every `levels` of them (half of that where it is even), so the first CTAs of
  // those with the most turns and of those with one less stand for all.
  const int pairs = (n + 1) / 2, g_pairs = pairs < sms ? pairs : sms, period = levels & 1 ? levels : levels / 2;
  const auto pairs_of = [&](int c) {
    int load = 0;
    for (int u = c; u < pairs; u += g_pairs)
      for (int k = 2 * u, pos = k % levels; k < 2 * u + 2 && k < n; ++k, pos = pos + 1 == levels ? 0 : pos + 1)
        load += work(pos & 1 ? levels - 1 - (pos >> 1) : pos >> 1);
    return load;
  };
  const int most_turns = (pairs - 1) % g_pairs + 1;
  for (int c = 0; c < most_turns && c < period; ++c) more(span.pairs, pairs_of(c));
  for (int c = most_turns; c < g_pairs && c < most_turns + period; ++c) more(span.pairs, pairs_of(c));
  // Longest first: along the CTAs the work of even rows falls and that of odd rows rises, so the longest CTA is the first
  // one, or one at which an odd row comes to a longer level.
  const int g = n < sms ? n : sms;
  const auto load_of = [&](int c) {
    int load = 0;
    for (int at = 0, r = 0; at < n; at += g, ++r)
      if (const int k = at + (r & 1 ? g - 1 - c : c); k < n) load += work(k / n_bh);
    return load;
  };
  span.longest_first = load_of(0);
  for (int at = g; at < n; at += 2 * g) {
    const int last = at + g < n ? at + g - 1 : n - 1;
    for (int level = at / n_bh; level <= last / n_bh; ++level) {
      const int k = (level + 1) * n_bh - 1;  // the last unit of this level
      more(span.longest_first, load_of(at + g - 1 - (k < last ? k : last)));
    }
  }
  return span;
}

// Kernels launched by this library since it was loaded (all devices, all threads).
extern std::atomic<uint64_t> g_kernel_launches;

// A launch answers with its own outcome: an error that an earlier call left behind is neither taken for it nor cleared.
template <typename Kern, typename Params>
inline int launch_counted(const cudaLaunchConfig_t& cfg, Kern kern, const Params& params) {
  if (cudaLaunchKernelEx(&cfg, kern, params) != cudaSuccess) return FA_ERR_CUDA;
  g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
  return FA_OK;
}

// Launch that starts when its predecessors on the stream are done.
template <typename Kern, typename Params>
inline int launch_ordered(Kern kern, dim3 grid, int threads, cudaStream_t stream, const Params& params) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  return launch_counted(cfg, kern, params);
}

// Launch with the programmatic-stream-serialization attribute (see grid_dep_wait()).
template <typename Kern, typename Params>
inline int launch_overlapped(Kern kern, dim3 grid, int threads, size_t smem, cudaStream_t stream,
                             const Params& params, int cluster_x = 1) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster_x;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster_x > 1 ? 2 : 1;
  return launch_counted(cfg, kern, params);
}

// Tile map for the slabs of a DsSlab: dims {N, M, problems, 1}, box {64, box_rows}.
inline int make_tmap_slab(CUtensorMap* out, const DsSlab& slab, int M, int N, int box_rows = 128) {
  const uint64_t dims[4] = {(uint64_t)N, (uint64_t)M, (uint64_t)slab.n_bh, 1};
  const uint64_t row = (uint64_t)slab.pitch * 2;
  const uint64_t sb[3] = {row, row * M, row * M * (uint64_t)slab.n_bh};
  const uint32_t box[4] = {64, (uint32_t)box_rows, 1, 1};
  return make_tmap_4d(out, slab.base, 2, dims, sb, box);
}

// What every entry point asks of a (B, S, H, D) operand, whether its kernel reads it through a tile map (whose
// encoding refuses the rest) or with plain loads: 16-byte aligned base and strides, no stride of zero or less.
inline bool operand_ok(const void* ptr, const int64_t s[3]) {
  return reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && s[0] > 0 && s[1] > 0 && s[2] > 0 && (s[0] | s[1] | s[2]) % 8 == 0;
}

// Head dims are computed on a padded width: 16/32/64 -> 64, 128 -> 128, 256 -> 256.
inline int padded_head_dim(int d) { return d <= 64 ? 64 : d; }

// Tile map for a (B, S, H, D) tensor: dims {D, H, S, B}, box {64, 1, rows, 1}.
inline int make_tmap_bshd(CUtensorMap* out, const void* base, int B, int S, int H, int D,
                          const int64_t stride[3], int box_rows) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  const uint64_t sb[3] = {(uint64_t)stride[2] * 2, (uint64_t)stride[1] * 2, (uint64_t)stride[0] * 2};
  const uint32_t box[4] = {64, 1, (uint32_t)box_rows, 1};
  return make_tmap_4d(out, base, 2, dims, sb, box);
}

// Tile map for a (B, S, H, D) result that leaves by bulk tensor stores of 32 rows and 64 columns.  False where the layout
// cannot be encoded, which plain stores can write to all the same (a stride of zero or less); the stride of a dimension of
// extent one does not matter.
inline bool make_tmap_result(CUtensorMap* out, const void* base, int B, int S, int H, int D, const int64_t stride[3]) {
  const int extent[3] = {B, S, H};
  int64_t s[3];
  for (int i = 0; i < 3; ++i) {
    s[i] = extent[i] == 1 ? 8 : stride[i];
    if (s[i] <= 0) return false;
  }
  return make_tmap_bshd(out, base, B, S, H, D, s, 32) == FA_OK;
}

// Tile map for a (B, H, M, N) bias-like tensor: dims {N, M, H, B}; a zero stride
// on B or H collapses that dimension to extent 1 (the kernel then passes
// coordinate 0).  box {box_cols, box_rows, 1, 1}.
inline int make_tmap_bhmn(CUtensorMap* out, const void* base, int elem_bytes, int B, int H, int M,
                          int N, const int64_t stride[3], int box_cols, int box_rows, int* b_mul,
                          int* h_mul) {
  const bool b0 = stride[0] == 0, h0 = stride[1] == 0;
  *b_mul = b0 ? 0 : 1;
  *h_mul = h0 ? 0 : 1;
  const uint64_t row_bytes = (uint64_t)stride[2] * elem_bytes;
  const uint64_t dims[4] = {(uint64_t)N, (uint64_t)M, (uint64_t)(h0 ? 1 : H), (uint64_t)(b0 ? 1 : B)};
  // a collapsed dimension still needs a legal (non-zero, 16-byte multiple) stride
  const uint64_t sb[3] = {row_bytes, h0 ? row_bytes * (uint64_t)M : (uint64_t)stride[1] * elem_bytes,
                          b0 ? row_bytes * (uint64_t)M : (uint64_t)stride[0] * elem_bytes};
  const uint32_t box[4] = {(uint32_t)box_cols, (uint32_t)box_rows, 1, 1};
  return make_tmap_4d(out, base, elem_bytes, dims, sb, box);
}

}  // namespace fa
