// Forward and backward for short sequences (windows, patches): M, N, D <= 64, one CTA per (batch, head).
//
// Such a problem is one tile for the 128-row kernels: 49 of 128 rows and keys of it used, a load, two or five products
// and an epilogue that nothing overlaps, and a backward of three launches with dS going through memory.  Here a CTA loads
// the whole problem into shared memory once, a warp takes 16 query rows, and the backward is one launch: delta, P and dS
// of all keys, dQ from the warp's own dS, then dK and dV by 16 keys a warp from P and dS in shared memory.  What bounds
// it is latency (loads, then a chain of a few hundred instructions), so many small CTAs per SM: four warps and 15 KB
// (forward) or 38 KB (backward) for a window of 49 x 49 and D = 32.  The warp-level matrix instruction is enough for that: a window has 16 rows a warp
// where tcgen05 wants 128, and a chain of its products would cost a round trip through tensor memory each.
// fp16, us, tile kernels -> here, forward and whole backward (without the copies of padded biases and gradients):
//   B256 H6 49 x 49 D32       no bias 32 -> 11, 52 -> 19     trained bias 41 -> 15, 58 -> 32     mask 42 -> 14, 60 -> 22
//   B256 H6 64 x 64 D64       no bias 31 -> 16, 60 -> 44     B1024 H12, trained bias 321 -> 127, 438 -> 453
//   (the one kind whose backward alone loses, up to 5 %: a trained 16-bit bias of each problem's own at D 64, 49 to 64 rows, thousands of
//   problems; forward and backward 1.3 times as fast.  1536 problems of 64 x 64: 40 -> 19, 65.0 -> 65.2; of 56 x 56: 41 -> 17, 64 -> 55)
//   B1024 H8 17 x 17 D16      trained bias 186 -> 24, 254 -> 51
// The limit is 64: with up to 128 rows and keys and eight warps the same kernels lost as soon as the problems fill the
// chip (B256 H12 128 x 128 D64: 57 -> 95, 152 -> 242; 96 x 96 D32, mask: 77 -> 74, 118 -> 159; 64 x 128: 53 -> 52,
// 123 -> 194), and a limit by the number of problems would make a head's result depend on the other heads of its call.
//
// Bias, mask and bias gradient are read and written element by element or by pairs, at any address and with any strides
// but the innermost, so neither needs a padded copy.
//
// Replaces _attn_fwd, _attn_bwd_preprocess, _attn_bwd_dkdv and _attn_bwd_dq of the reference (flash_attention.py 12-646)
// for short sequences: same masks, base-2 softmax, log-sum-exp, dbias = dS.
#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

struct SmallParams {
  const void* q;
  const void* k;
  const void* v;
  const void* bias;
  void* o;     // forward: out; backward: in
  float* lse;  // forward: out; backward: in
  const void* d_o;
  void* dq;
  void* dk;
  void* dv;
  void* dbias;  // backward: gradient of a 16-bit or fp32 bias, or null
  void* ds16;   // backward with an fp32 bias: where a caller wants dS in 16 bits as well, or null
  float* delta;
  int* status;
  int64_t q_sB, q_sM, q_sH, k_sB, k_sN, k_sH, v_sB, v_sN, v_sH, o_sB, o_sM, o_sH;
  int64_t do_sB, do_sM, do_sH, dq_sB, dq_sM, dq_sH, dk_sB, dk_sN, dk_sH, dv_sB, dv_sN, dv_sH;
  int64_t bias_sB, bias_sH, bias_sM, db_sB, db_sH, db_sM, ds_sB, ds_sH, ds_sM;
  int H, M, N;
  int causal;
  int bias_pairs, db_pairs;  // two neighbouring elements (of an even column) may be accessed at once: N and strides are even
  float sm_scale;
};

template <typename T>
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if constexpr (Pack2<T>::kIsBf16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// Row-major tiles in shared memory: 16 bytes between rows keep the eight rows of an ldmatrix tile in different banks.
template <int D>
constexpr int kPitch = D * 2 + 16;

// Rows 0 .. rows-1 of a (S, D) operand; zeros up to a multiple of 16 rows.  Asynchronous, so that all of a CTA's loads travel
// together (through registers, a loop of load and store per 16 bytes, a 128-row problem took 4 us longer).
template <int D>
__device__ __forceinline__ void load_rows(uint32_t dst, const void* src, int64_t stride, int rows) {
  constexpr int C = D / 8;  // 16-byte chunks of a row
  const int all = (rows + 15) / 16 * 16 * C;
  for (int i = threadIdx.x; i < all; i += blockDim.x) {
    const int r = i / C, c = i % C;
    const void* from = static_cast<const uint16_t*>(src) + min(r, rows - 1) * stride + c * 8;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * kPitch<D> + c * 16), "l"(from),
                 "r"(r < rows ? 16 : 0)
                 : "memory");
  }
}
__device__ __forceinline__ void loads_landed() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// The bias of rows r, r + 8 and columns c, c + 1 of the eight groups of 8 keys: 16-bit pairs, bytes (one each
// half word) or fp32 values.  All loads are issued at once, from clamped places (what lies beyond M or N is not used).
template <int BIAS>
struct BiasFrag {
  uint32_t w[BIAS == 3 ? 32 : (BIAS == 0 ? 1 : 16)];
};
template <int BIAS>
__device__ __forceinline__ void load_bias(BiasFrag<BIAS>& f, const SmallParams& p, int64_t off, int r, int c) {
#pragma unroll
  for (int hf = 0; BIAS != 0 && hf < 2; ++hf) {
    const int64_t row = off + min(r + hf * 8, p.M - 1) * p.bias_sM;
    if (BIAS == 1 && p.bias_pairs) {  // (N is even)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        f.w[hf * 8 + i] = __ldcg(reinterpret_cast<const uint32_t*>(static_cast<const uint16_t*>(p.bias) + row + min(i * 8 + c, p.N - 2)));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int64_t a = row + min(i * 8 + c, p.N - 1), b = row + min(i * 8 + c + 1, p.N - 1);
        if constexpr (BIAS == 1) {
          const uint16_t* src = static_cast<const uint16_t*>(p.bias);
          f.w[hf * 8 + i] = __ldcg(src + a) | static_cast<uint32_t>(__ldcg(src + b)) << 16;
        } else if constexpr (BIAS == 2) {
          const uint8_t* src = static_cast<const uint8_t*>(p.bias);
          f.w[hf * 8 + i] = __ldcg(src + a) | static_cast<uint32_t>(__ldcg(src + b)) << 16;
        } else {
          const uint32_t* src = static_cast<const uint32_t*>(p.bias);
          f.w[(hf * 8 + i) * 2] = __ldcg(src + a);
          f.w[(hf * 8 + i) * 2 + 1] = __ldcg(src + b);
        }
      }
    }
  }
}
// Group i, row half hf: two biases in natural units, or a mask as 0 (seen) and -inf.
template <int BIAS, typename T>
__device__ __forceinline__ float2 bias_pair(const BiasFrag<BIAS>& f, int i, int hf) {
  if constexpr (BIAS == 1) return Pack2<T>::unpack(f.w[hf * 8 + i]);
  if constexpr (BIAS == 2) return make_float2(f.w[hf * 8 + i] & 0xFFFFu ? 0.f : -INFINITY, f.w[hf * 8 + i] >> 16 ? 0.f : -INFINITY);
  return make_float2(__uint_as_float(f.w[(hf * 8 + i) * 2]), __uint_as_float(f.w[(hf * 8 + i) * 2 + 1]));
}

// S = Q K^T of 16 query rows (fragments `qa`): s[i] is the i-th group of 8 keys.
template <int D, typename T>
__device__ __forceinline__ void product_nt(float (*s)[4], const uint32_t (*qa)[4], uint32_t k_tile, int n_keys, int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[i][e] = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // 16 keys at a time
    const int n0 = i * 16;
    if (n0 >= n_keys) break;
    const uint32_t row = k_tile + (n0 + (lane & 7) + ((lane >> 4) << 3)) * kPitch<D> + ((lane >> 3) & 1) * 16;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      uint32_t b[4];
      ldsm4(row + ks * 32, b);
      mma16816<T>(s[2 * i], qa[ks], b[0], b[1]);
      mma16816<T>(s[2 * i + 1], qa[ks], b[2], b[3]);
    }
  }
}
// acc[16 rows][D] += A[16 rows][16] B[16][D], B row-major in shared memory from row `r0` on.
template <int D, typename T>
__device__ __forceinline__ void product_nn(float (*acc)[4], const uint32_t* a, uint32_t b_tile, int r0, int lane) {
  const uint32_t row = b_tile + (r0 + (lane & 15)) * kPitch<D> + (lane >> 4) * 16;
#pragma unroll
  for (int j = 0; j < D / 16; ++j) {
    uint32_t b[4];
    ldsm4_trans(row + j * 32, b);
    mma16816<T>(acc[2 * j], a, b[0], b[1]);
    mma16816<T>(acc[2 * j + 1], a, b[2], b[3]);
  }
}
// The 16 x D result of a warp, rows r and r + 8 of each lane's quad.
template <int D, typename T>
__device__ __forceinline__ void store_rows(T* out, int64_t stride, const float (*acc)[4], float mul0, float mul1, int r, int rows, int c) {
#pragma unroll
  for (int j = 0; j < D / 8; ++j) {
    if (r < rows)
      *reinterpret_cast<uint32_t*>(out + r * stride + j * 8 + c) = Pack2<T>::pack(acc[j][0] * mul0, acc[j][1] * mul0);
    if (r + 8 < rows)
      *reinterpret_cast<uint32_t*>(out + (r + 8) * stride + j * 8 + c) = Pack2<T>::pack(acc[j][2] * mul1, acc[j][3] * mul1);
  }
}
template <int D>
__device__ __forceinline__ void load_a(uint32_t (*a)[4], uint32_t tile, int r0, int lane) {
  const uint32_t row = tile + (r0 + (lane & 15)) * kPitch<D> + (lane >> 4) * 16;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) ldsm4(row + ks * 32, a[ks]);
}

template <int D, typename T, int BIAS>
__global__ void __launch_bounds__(128) small_fwd_kernel(const SmallParams p) {
  using P2 = Pack2<T>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.x, b = bh / p.H, h = bh - b * p.H;
  const int m_pad = (p.M + 15) / 16 * 16, n_pad = (p.N + 15) / 16 * 16;
  const uint32_t sq = smem_u32(smem_raw), sk = sq + m_pad * kPitch<D>, sv = sk + n_pad * kPitch<D>;
  grid_dep_launch_next();
  grid_dep_wait();  // the previous kernel's results (and the status word) are visible from here
  if (*reinterpret_cast<volatile int*>(p.status) != 0) return;
  load_rows<D>(sq, static_cast<const T*>(p.q) + b * p.q_sB + h * p.q_sH, p.q_sM, p.M);
  load_rows<D>(sk, static_cast<const T*>(p.k) + b * p.k_sB + h * p.k_sH, p.k_sN, p.N);
  load_rows<D>(sv, static_cast<const T*>(p.v) + b * p.v_sB + h * p.v_sH, p.v_sN, p.N);
  const int m0 = warp * 16;
  const int r = m0 + (lane >> 2), c = (lane & 3) * 2;  // this lane's rows r, r + 8 and columns c, c + 1 of every eight
  const int64_t bias0 = b * p.bias_sB + h * p.bias_sH;
  BiasFrag<BIAS> bias;
  load_bias<BIAS>(bias, p, bias0, r, c);
  loads_landed();
  if (m0 >= p.M) return;

  uint32_t qa[D / 16][4];
  load_a<D>(qa, sq, m0, lane);
  const float scale_log2 = p.sm_scale * kLog2e;
  float s[8][4];
  float mx[2] = {-INFINITY, -INFINITY};
  product_nt<D, T>(s, qa, sk, p.N, lane);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int n = i * 8 + c;
    float* x = s[i];
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] *= scale_log2;
    if constexpr (BIAS != 0) {
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const float2 f = bias_pair<BIAS, T>(bias, i, hf);
        if (BIAS == 2) {
          if (f.x != 0.f) x[hf * 2] = -INFINITY;
          if (f.y != 0.f) x[hf * 2 + 1] = -INFINITY;
        } else {
          x[hf * 2] = fmaf(f.x, kLog2e, x[hf * 2]);
          x[hf * 2 + 1] = fmaf(f.y, kLog2e, x[hf * 2 + 1]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = r + (e >> 1) * 8, nn = n + (e & 1);
      if (nn >= p.N || (p.causal && nn > m)) x[e] = -INFINITY;
      mx[e >> 1] = fmaxf(mx[e >> 1], x[e]);
    }
  }
  float l[2];
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    mx[hf] = fmaxf(mx[hf], __shfl_xor_sync(0xffffffffu, mx[hf], 1));
    mx[hf] = fmaxf(mx[hf], __shfl_xor_sync(0xffffffffu, mx[hf], 2));
    const float neg_m = mx[hf] == -INFINITY ? 0.f : -mx[hf];
    l[hf] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[i][hf * 2 + e] = ex2(s[i][hf * 2 + e] + neg_m);
        l[hf] += s[i][hf * 2 + e];
      }
    l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 1);
    l[hf] += __shfl_xor_sync(0xffffffffu, l[hf], 2);
  }
  float o[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k * 16 >= p.N) break;
    const uint32_t a[4] = {P2::pack(s[2 * k][0], s[2 * k][1]), P2::pack(s[2 * k][2], s[2 * k][3]),
                           P2::pack(s[2 * k + 1][0], s[2 * k + 1][1]), P2::pack(s[2 * k + 1][2], s[2 * k + 1][3])};
    product_nn<D, T>(o, a, sv, k * 16, lane);
  }
  // a row whose keys are all masked out: output 0, LSE +inf
  float inv[2];
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    const bool any_key = mx[hf] != -INFINITY && l[hf] > 0.f;
    inv[hf] = any_key ? 1.0f / l[hf] : 0.f;
    const int m = r + hf * 8;
    if ((lane & 3) == 0 && m < p.M) p.lse[static_cast<int64_t>(bh) * p.M + m] = any_key ? mx[hf] + log2f(l[hf]) : INFINITY;
  }
  store_rows<D, T>(static_cast<T*>(p.o) + b * p.o_sB + h * p.o_sH, p.o_sM, o, inv[0], inv[1], r, p.M, c);
}

// DS16: dS goes out in 16 bits besides.  A variant of its own: asked for at run time it made the calls that do not want it
// slower (fp32 bias, B256 H6 49 x 49 D32 26.5 -> 27.9 us, B1024 H8 17 x 17 D16 30.2 -> 32.2).
template <int D, typename T, int BIAS, bool DS16 = false>
__global__ void __launch_bounds__(128) small_bwd_kernel(const SmallParams p) {
  using P2 = Pack2<T>;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.x, b = bh / p.H, h = bh - b * p.H;
  const int m_pad = (p.M + 15) / 16 * 16, n_pad = (p.N + 15) / 16 * 16;
  const int pitch = n_pad * 2 + 16;  // of a row of P or dS
  const uint32_t sq = smem_u32(smem_raw), sdo = sq + m_pad * kPitch<D>, sk = sdo + m_pad * kPitch<D>;
  const uint32_t sv = sk + n_pad * kPitch<D>, sp = sv + n_pad * kPitch<D>, sds = sp + m_pad * pitch;
  grid_dep_launch_next();
  grid_dep_wait();  // the previous kernels' results (and the status word) are visible from here
  if (*reinterpret_cast<volatile int*>(p.status) != 0) return;
  load_rows<D>(sq, static_cast<const T*>(p.q) + b * p.q_sB + h * p.q_sH, p.q_sM, p.M);
  load_rows<D>(sdo, static_cast<const T*>(p.d_o) + b * p.do_sB + h * p.do_sH, p.do_sM, p.M);
  load_rows<D>(sk, static_cast<const T*>(p.k) + b * p.k_sB + h * p.k_sH, p.k_sN, p.N);
  load_rows<D>(sv, static_cast<const T*>(p.v) + b * p.v_sB + h * p.v_sH, p.v_sN, p.N);
  const int m0 = warp * 16;
  const int r = m0 + (lane >> 2), c = (lane & 3) * 2;
  const int64_t bias0 = b * p.bias_sB + h * p.bias_sH;
  BiasFrag<BIAS> bias;
  load_bias<BIAS>(bias, p, bias0, r, c);
  // -LSE2 and -delta of rows r and r + 8; delta = rowsum(o * do), two lanes a row.  Rows beyond M get -inf / 0, which makes
  // their P and dS zero.
  float nl[2], nd[2];
  {
    float acc = 0.f;
    const int m = m0 + (lane >> 1);
    if (m < p.M) {
      constexpr int C = D / 16;  // 16-byte chunks of half a row
      const uint4* orow = reinterpret_cast<const uint4*>(static_cast<const T*>(p.o) + b * p.o_sB + h * p.o_sH + m * p.o_sM) + (lane & 1) * C;
      const uint4* grow = reinterpret_cast<const uint4*>(static_cast<const T*>(p.d_o) + b * p.do_sB + h * p.do_sH + m * p.do_sM) + (lane & 1) * C;
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const uint4 x = __ldcg(orow + i), y = __ldcg(grow + i);
        const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 u = P2::unpack(xw[e]), w = P2::unpack(yw[e]);
          acc = fmaf(u.x, w.x, acc);
          acc = fmaf(u.y, w.y, acc);
        }
      }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    if ((lane & 1) == 0 && m < p.M) p.delta[static_cast<int64_t>(bh) * p.M + m] = acc;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const float d = __shfl_sync(0xffffffffu, acc, ((lane >> 2) + hf * 8) * 2);
      const int row = r + hf * 8;
      nl[hf] = row < p.M ? -__ldcg(p.lse + static_cast<int64_t>(bh) * p.M + row) : -INFINITY;
      nd[hf] = row < p.M ? -d : 0.f;
    }
  }
  loads_landed();

  // ---- 16 query rows a warp: P and dS, the bias gradient, dQ
  if (m0 < p.M) {
    uint32_t qa[D / 16][4], ga[D / 16][4];
    load_a<D>(qa, sq, m0, lane);
    load_a<D>(ga, sdo, m0, lane);
    const float scale_log2 = p.sm_scale * kLog2e;
    float dq[D / 8][4];
#pragma unroll
    for (int j = 0; j < D / 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) dq[j][e] = 0.f;
    float s[8][4], g[8][4];
    product_nt<D, T>(s, qa, sk, p.N, lane);
    product_nt<D, T>(g, ga, sv, p.N, lane);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int n = i * 8 + c;
      if (i * 8 >= n_pad) break;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int m = r + hf * 8;
        float x[2] = {fmaf(s[i][hf * 2], scale_log2, nl[hf]), fmaf(s[i][hf * 2 + 1], scale_log2, nl[hf])};
        bool keep[2] = {n < p.N && m < p.M, n + 1 < p.N && m < p.M};
        if constexpr (BIAS != 0) {
          const float2 f = bias_pair<BIAS, T>(bias, i, hf);
          if (BIAS == 2) {
            keep[0] = keep[0] && f.x == 0.f;
            keep[1] = keep[1] && f.y == 0.f;
          } else {
            x[0] = fmaf(f.x, kLog2e, x[0]);
            x[1] = fmaf(f.y, kLog2e, x[1]);
          }
        }
        if (p.causal) {
          keep[0] = keep[0] && n <= m;
          keep[1] = keep[1] && n + 1 <= m;
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float pe = keep[e] ? ex2(x[e]) : 0.f;
          s[i][hf * 2 + e] = pe;
          g[i][hf * 2 + e] = n + e < p.N ? pe * (g[i][hf * 2 + e] + nd[hf]) : 0.f;
        }
        const uint32_t d2 = P2::pack(g[i][hf * 2], g[i][hf * 2 + 1]);
        const uint32_t off = m * pitch + n * 2;
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sp + off), "r"(P2::pack(s[i][hf * 2], s[i][hf * 2 + 1])) : "memory");
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(sds + off), "r"(d2) : "memory");
        if (BIAS == 3 && p.dbias != nullptr && m < p.M && n < p.N) {  // the fp32 gradient goes out unrounded
          float* dst = static_cast<float*>(p.dbias) + b * p.db_sB + h * p.db_sH + m * p.db_sM + n;
          dst[0] = g[i][hf * 2];
          if (n + 1 < p.N) dst[1] = g[i][hf * 2 + 1];
        }
        if constexpr (DS16) {
          if (m < p.M && n < p.N) {  // (rows start at multiples of 16 bytes, n is even)
            uint16_t* dst = static_cast<uint16_t*>(p.ds16) + b * p.ds_sB + h * p.ds_sH + m * p.ds_sM + n;
            if (n + 1 < p.N)
              *reinterpret_cast<uint32_t*>(dst) = d2;
            else
              *dst = static_cast<uint16_t>(d2);
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k * 16 >= n_pad) break;
      const uint32_t a[4] = {P2::pack(g[2 * k][0], g[2 * k][1]), P2::pack(g[2 * k][2], g[2 * k][3]),
                             P2::pack(g[2 * k + 1][0], g[2 * k + 1][1]), P2::pack(g[2 * k + 1][2], g[2 * k + 1][3])};
      product_nn<D, T>(dq, a, sk, k * 16, lane);
    }
    if (BIAS == 1 && p.dbias != nullptr) {
      // the warp's rows of dS, whole rows at a time
      __syncwarp();
      uint16_t* dst = static_cast<uint16_t*>(p.dbias) + b * p.db_sB + h * p.db_sH + m0 * p.db_sM;
      const uint32_t from = sds + m0 * pitch;
      const int rows = min(16, p.M - m0);
#pragma unroll 4
      for (int i = 0; i < rows; ++i) {
        if (p.db_pairs) {  // (N is even)
          for (int n = lane * 2; n < p.N; n += 64) {
            uint32_t v;
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(from + i * pitch + n * 2) : "memory");
            *reinterpret_cast<uint32_t*>(dst + n) = v;
          }
        } else {
          for (int n = lane; n < p.N; n += 32) {
            uint16_t v;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(from + i * pitch + n * 2) : "memory");
            dst[n] = v;
          }
        }
        dst += p.db_sM;
      }
    }
    store_rows<D, T>(static_cast<T*>(p.dq) + b * p.dq_sB + h * p.dq_sH, p.dq_sM, dq, p.sm_scale, p.sm_scale, r, p.M, c);
  }
  __syncthreads();

  // ---- 16 keys a warp: dV = P^T dO, dK = sm_scale * dS^T Q
  const int n0 = warp * 16;
  if (n0 >= p.N) return;
  float dv[D / 8][4], dk[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) dv[j][e] = dk[j][e] = 0.f;
  // transposed 16 x 16 operand: tiles (rows m 0-7 / 8-15) x (keys 0-7 / 8-15)
  const uint32_t at = ((lane & 7) + ((lane >> 4) << 3)) * pitch + (n0 + ((lane >> 3) & 1) * 8) * 2;
  const int first = p.causal ? n0 : 0;  // query rows above the keys see none of them
#pragma unroll 2
  for (int mk = first; mk < m_pad; mk += 16) {
    uint32_t a[4];
    ldsm4_trans(sp + at + mk * pitch, a);
    product_nn<D, T>(dv, a, sdo, mk, lane);
    ldsm4_trans(sds + at + mk * pitch, a);
    product_nn<D, T>(dk, a, sq, mk, lane);
  }
  const int n = n0 + (lane >> 2);
  store_rows<D, T>(static_cast<T*>(p.dv) + b * p.dv_sB + h * p.dv_sH, p.dv_sN, dv, 1.f, 1.f, n, p.N, c);
  store_rows<D, T>(static_cast<T*>(p.dk) + b * p.dk_sB + h * p.dk_sH, p.dk_sN, dk, p.sm_scale, p.sm_scale, n, p.N, c);
}

template <typename K>
int configure(K kern, int bytes, bool* configured) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return FA_ERR_CUDA;
    configured[dev] = true;
  }
  return FA_OK;
}

constexpr int fwd_bytes(int D, int m, int n) { return (m + 2 * n) * (D * 2 + 16); }
constexpr int bwd_bytes(int D, int m, int n) { return 2 * (m + n) * (D * 2 + 16) + 2 * m * (n * 2 + 16); }

template <int D, typename T, int BIAS>
int launch_inst(const SmallParams& sp, int bh, bool bwd, cudaStream_t stream) {
  static bool set_fwd[64] = {}, set_bwd[64] = {};
  const int m = (sp.M + 15) / 16 * 16, n = (sp.N + 15) / 16 * 16;
  const int warps = (bwd && n > m ? n : m) / 16;
  if constexpr (BIAS == 3) {
    if (bwd && sp.ds16 != nullptr) {
      static bool set_ds16[64] = {};
      auto kern = small_bwd_kernel<D, T, BIAS, true>;
      if (int r = configure(kern, bwd_bytes(D, 64, 64), set_ds16)) return r;
      return launch_overlapped(kern, dim3(bh), warps * 32, bwd_bytes(D, m, n), stream, sp);
    }
  }
  if (bwd) {
    auto kern = small_bwd_kernel<D, T, BIAS>;
    if (int r = configure(kern, bwd_bytes(D, 64, 64), set_bwd)) return r;
    return launch_overlapped(kern, dim3(bh), warps * 32, bwd_bytes(D, m, n), stream, sp);
  }
  auto kern = small_fwd_kernel<D, T, BIAS>;
  if (int r = configure(kern, fwd_bytes(D, 64, 64), set_fwd)) return r;
  return launch_overlapped(kern, dim3(bh), warps * 32, fwd_bytes(D, m, n), stream, sp);
}

template <int D, typename T>
int launch_bias(const SmallParams& sp, int bias_kind, int bh, bool bwd, cudaStream_t stream) {
  switch (bias_kind) {
    case FA_BIAS_NONE: return launch_inst<D, T, 0>(sp, bh, bwd, stream);
    case FA_BIAS_SAME: return launch_inst<D, T, 1>(sp, bh, bwd, stream);
    case FA_BIAS_BOOL: return launch_inst<D, T, 2>(sp, bh, bwd, stream);
    case FA_BIAS_F32: return launch_inst<D, T, 3>(sp, bh, bwd, stream);
    default: return FA_ERR_UNSUPPORTED;
  }
}
template <typename T>
int launch_dim(const SmallParams& sp, int D, int bias_kind, int bh, bool bwd, cudaStream_t stream) {
  return D == 16   ? launch_bias<16, T>(sp, bias_kind, bh, bwd, stream)
         : D == 32 ? launch_bias<32, T>(sp, bias_kind, bh, bwd, stream)
                   : launch_bias<64, T>(sp, bias_kind, bh, bwd, stream);
}

bool pairs_ok(const void* ptr, const int64_t* s, int N) {
  return N % 2 == 0 && reinterpret_cast<uintptr_t>(ptr) % 4 == 0 && (s[0] | s[1] | s[2]) % 2 == 0;
}

}  // namespace

bool small_takes(int M, int N, int D) { return M <= 64 && N <= 64 && D <= 64; }

int check_tiled_bias(const fa_params& p, bool bwd) {
  const auto bad = [](const void* ptr, const int64_t* s, int eb) {
    return reinterpret_cast<uintptr_t>(ptr) % 16 != 0 || s[0] < 0 || s[1] < 0 || s[2] <= 0 || (s[0] * eb) % 16 || (s[1] * eb) % 16 ||
           (s[2] * eb) % 16;
  };
  const auto real = [](const int64_t* s) { return s[0] > 0 && s[1] > 0; };  // not expanded
  const bool f32 = p.bias_kind == FA_BIAS_F32;
  const int eb = p.bias_kind == FA_BIAS_BOOL ? 1 : (f32 ? 4 : 2);
  if (p.bias_kind != FA_BIAS_NONE && bad(p.bias, p.bias_stride, eb)) return FA_ERR_ALIGN;
  if (!bwd) return FA_OK;
  if (p.write_dbias && (bad(p.dbias, p.dbias_stride, eb) || !real(p.dbias_stride))) return FA_ERR_ALIGN;
  if (f32 && p.ds16 && (bad(p.ds16, p.ds16_stride, 2) || !real(p.ds16_stride))) return FA_ERR_ALIGN;
  return FA_OK;
}

int launch_small(const fa_params& p, bool bwd, cudaStream_t stream, int* status) {
  auto bad = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 16 != 0 || s[0] % 8 || s[1] % 8 || s[2] % 8;
  };
  if (!operand_ok(p.q, p.q_stride) || !operand_ok(p.k, p.k_stride) || !operand_ok(p.v, p.v_stride) || bad(p.o, p.o_stride))
    return FA_ERR_ALIGN;
  SmallParams s = {};
  s.q = p.q, s.k = p.k, s.v = p.v, s.bias = p.bias, s.o = p.o, s.lse = p.lse, s.status = status;
  s.q_sB = p.q_stride[0], s.q_sM = p.q_stride[1], s.q_sH = p.q_stride[2];
  s.k_sB = p.k_stride[0], s.k_sN = p.k_stride[1], s.k_sH = p.k_stride[2];
  s.v_sB = p.v_stride[0], s.v_sN = p.v_stride[1], s.v_sH = p.v_stride[2];
  s.o_sB = p.o_stride[0], s.o_sM = p.o_stride[1], s.o_sH = p.o_stride[2];
  s.bias_sB = p.bias_stride[0], s.bias_sH = p.bias_stride[1], s.bias_sM = p.bias_stride[2];
  s.bias_pairs = p.bias_kind == FA_BIAS_SAME && pairs_ok(p.bias, p.bias_stride, p.N);
  s.H = p.H, s.M = p.M, s.N = p.N;
  s.causal = p.causal ? 1 : 0;
  s.sm_scale = p.sm_scale;
  if (bwd) {
    if (!operand_ok(p.d_o, p.do_stride) || bad(p.dq, p.dq_stride) || bad(p.dk, p.dk_stride) || bad(p.dv, p.dv_stride))
      return FA_ERR_ALIGN;
    s.d_o = p.d_o, s.dq = p.dq, s.dk = p.dk, s.dv = p.dv, s.delta = p.delta;
    s.do_sB = p.do_stride[0], s.do_sM = p.do_stride[1], s.do_sH = p.do_stride[2];
    s.dq_sB = p.dq_stride[0], s.dq_sM = p.dq_stride[1], s.dq_sH = p.dq_stride[2];
    s.dk_sB = p.dk_stride[0], s.dk_sN = p.dk_stride[1], s.dk_sH = p.dk_stride[2];
    s.dv_sB = p.dv_stride[0], s.dv_sN = p.dv_stride[1], s.dv_sH = p.dv_stride[2];
    if (p.write_dbias) {
      s.dbias = p.dbias;
      s.db_sB = p.dbias_stride[0], s.db_sH = p.dbias_stride[1], s.db_sM = p.dbias_stride[2];
      s.db_pairs = p.bias_kind == FA_BIAS_SAME && pairs_ok(p.dbias, p.dbias_stride, p.N);
    }
    if (p.bias_kind == FA_BIAS_F32) {
      s.ds16 = p.ds16;
      s.ds_sB = p.ds16_stride[0], s.ds_sH = p.ds16_stride[1], s.ds_sM = p.ds16_stride[2];
    }
  }
  const int bh = p.B * p.H;
  return p.dtype == FA_BF16 ? launch_dim<__nv_bfloat16>(s, p.D, p.bias_kind, bh, bwd, stream)
                            : launch_dim<__half>(s, p.D, p.bias_kind, bh, bwd, stream);
}

}  // namespace fa
