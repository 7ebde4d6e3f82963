// Forward attention for a handful of query rows (decoding: one or a few new tokens against a long
// key / value cache) on sm_100a.
//
// With M <= 16 the path is a stream over K and V: 2 N D elements are read once and each takes part in
// at most 16 multiply-adds, a few per cent of what the 128-row tile kernel would spend on its
// padding.  What matters is bytes in flight, so K and V go straight from global memory into
// registers in the layout the warp-level matrix instruction wants (no shared memory, no barriers),
// one 16-key tile ahead, and the keys of a (batch, head) are spread over all warps of a cluster
// of CTAs, so that even a few heads fill the chip.  (The tile kernel gives each head to one CTA.)
// The warp-level matrix instruction is enough: at the HBM rate an SM has 350 cycles for the 32 products
// of a tile, and tcgen05 would want the operands in shared memory and 128 rows of queries.
//   tile kernel -> here, bf16, us:  B8 H32 N4096 D128, M=1 120 -> 93 (5.8 TB/s), M=16 119 -> 115;  B1 H32 N20011
//   277 -> 60;  B64 H32 N2048 407 -> 325 (6.6 TB/s);  B32 H32 N1000 D64 92 -> 57.  A ring of asynchronous copies in shared memory in place of the
//   register tiles, two or three tiles deep, was slower (109 and 71 us for the first two).
//
// Per warp and tile of 16 keys (r = lane / 4, t = lane % 4):
//   S^T [16 keys x 8 queries] = K Q^T    the four lanes of a row load 16 bytes each: 64 contiguous
//        bytes of a key.  Which of the loaded elements meet in one k16 step is free as long as Q is
//        read the same way, so the words of a 16-byte load feed two steps.
//   P^T = exp2(S^T - m), transposed in registers (movmatrix) into the B operand
//   O^T [D x 8 queries] += V^T P^T       lane r loads elements 8r .. 8r+7 of keys 2t, 2t+1, 2t+8, 2t+9
//        (eight lanes: 128 contiguous bytes) and pairs the keys with byte permutes.
// The running maximum is raised only when some score passes it by more than 8 (log2 units), so the
// common tile needs one vote and no shuffles; row sums stay per lane until the end.
// A result must not depend on how many heads a call has, although the split over warps and CTAs does.  So the
// keys of a head are cut into leaves of a few tiles, by their number alone: a leaf has its own running maximum
// and starts from zero, four leaves in a row are folded from left to right into a group, and the groups (at most
// 32) are summed in order.  Whoever computes or folds a leaf, the operations and their order are the same.  A warp
// keeps its partial results in shared memory, whole groups or, where the heads are too few for that, leaves;
// the CTA folds those, and the cluster sums the groups through distributed shared memory.
//
// Replaces _attn_fwd of the reference (flash_attention.py 12-194) for short queries: same masks,
// bias, base-2 softmax and log-sum-exp as the tile kernel.
#include <cooperative_groups.h>

#include <mutex>

#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

namespace cg = cooperative_groups;

struct DecodeParams {
  const void* q;
  const void* k;
  const void* v;
  const void* bias;
  void* o;
  float* lse;
  int* status;
  int64_t q_sB, q_sM, q_sH, k_sB, k_sN, k_sH, v_sB, v_sN, v_sH, o_sB, o_sM, o_sH;
  int64_t bias_sB, bias_sH, bias_sM;
  int H, M, N, D;
  int n_keys;  // keys some row sees: N, or min(N, M) when causal
  int leaf;    // tiles of 16 keys in a leaf
  int fold;    // leaves in a partial result that a warp keeps: 1 or kGroup
  int own;     // partial results of a warp
  int causal;
  float sm_scale;
};

__device__ __forceinline__ uint4 ldg_stream(const void* ptr, bool ok) {
  uint4 v = make_uint4(0, 0, 0, 0);
  if (ok)
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(ptr));
  return v;
}

template <typename T>
__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  if constexpr (Pack2<T>::kIsBf16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// The bias of one score; a mask as 1 (seen) or 0.
template <int BIAS, typename T>
__device__ __forceinline__ float load_bias(const DecodeParams& p, int64_t off) {
  if constexpr (BIAS == 1) return static_cast<float>(static_cast<const T*>(p.bias)[off]);
  if constexpr (BIAS == 2) return static_cast<const uint8_t*>(p.bias)[off] ? 1.f : 0.f;
  if constexpr (BIAS == 3) return static_cast<const float*>(p.bias)[off];
  return 0.f;
}

constexpr int kGroup = 4;       // leaves in a group
constexpr int kMaxGroups = 32;  // of a head
constexpr int kMaxLeaves = kGroup * kMaxGroups;

// The shared memory of a CTA: room for the partial results of its warps, 16 rows for each group of 8 query rows a warp.
// What is not shared memory buffers the loads in flight, as much again: with twice the room B8 H32 N4096 D128 took
// 174 us instead of 90.
template <int DP, int NQ, int W>
struct DecodeSmem {
  static constexpr int kRows = 16 * NQ;   // query rows of partial results that a warp has room for
  static constexpr int kRow = DP + 8;     // accumulators of a row, and its sum in eight parts (one per lane that has it)
  float o[W * kRows * kRow];              // [partial result][query row][kRow]
  float m[W * kRows], gm[W * kRows];      // maximum of a partial result's row; the same of a group, at its first leaf
  float weight[NQ * 8][kMaxGroups];
  float m_all[NQ * 8], l_all[NQ * 8];
  const float* group[kMaxGroups];  // accumulators of a group, wherever in the cluster they are
  // partial results that a warp has room for; more than 8 would not make a better split
  static constexpr int slots(int rows) { return kRows / rows < 8 ? kRows / rows : 8; }
};

// What a partial result with maximum m counts in one with maximum m_all >= m; 0 where it has no key (its accumulators
// are zero then, or NaN, which stays).
__device__ __forceinline__ float weight_of(float m, float m_all) { return m == -INFINITY ? 0.f : ex2(m - m_all); }

// acc, of weight fa, followed by x, of weight fx.  (Spelled out, so that every place that folds rounds alike.)
__device__ __forceinline__ float fold2(float fa, float acc, float fx, float x) {
  return __fmaf_rn(fx, x, __fmul_rn(fa, acc));
}

// CTAs per SM: what the registers of the tile loop allow (a few words spill with a bias).
constexpr int decode_ctas(int DP, int NQ, int W) { return (DP == 64 ? (NQ == 1 ? 20 : 16) : (NQ == 1 ? 12 : 8)) / W; }

// DP: head dim rounded up to 64 or 128; NQ: groups of 8 query rows; W: warps per CTA.
// Grid: (cluster size, B * H).  The CTAs of a cluster share one (batch, head).
template <int DP, int NQ, int W, typename T, int BIAS>
__global__ void __launch_bounds__(W * 32, decode_ctas(DP, NQ, W)) decode_kernel(const DecodeParams p) {
  using P2 = Pack2<T>;
  using Smem = DecodeSmem<DP, NQ, W>;
  constexpr int KG = DP / 32;  // 16-byte loads per lane and key row of K
  constexpr int VG = DP / 64;  // ... of V

  extern __shared__ __align__(16) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = lane >> 2, t = lane & 3;
  const int bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
  grid_dep_launch_next();
  grid_dep_wait();  // the previous kernel's results (and the status word) are visible from here
  const bool live = *reinterpret_cast<volatile int*>(p.status) == 0;

  const int n_tiles = live ? (p.n_keys + 15) >> 4 : 0;
  const int first = (static_cast<int>(blockIdx.x) * W + warp) * p.own * p.fold * p.leaf;
  const int last = min(first + p.own * p.fold * p.leaf, n_tiles);

  // Q as the B operand: row = query, the same 16-byte pieces of the head dim as a key's
  uint4 q[NQ][KG];
  const T* qb = static_cast<const T*>(p.q) + b * p.q_sB + h * p.q_sH;
#pragma unroll
  for (int n = 0; n < NQ; ++n)
#pragma unroll
    for (int g = 0; g < KG; ++g) {
      const int m = n * 8 + r, d = g * 32 + t * 8;
      q[n][g] = m < p.M && d < p.D ? __ldcg(reinterpret_cast<const uint4*>(qb + m * p.q_sM + d)) : make_uint4(0, 0, 0, 0);
    }

  const T* kb = static_cast<const T*>(p.k) + b * p.k_sB + h * p.k_sH + t * 8;
  const T* vb = static_cast<const T*>(p.v) + b * p.v_sB + h * p.v_sH + r * 8;
  const int64_t bias_bh = b * p.bias_sB + h * p.bias_sH;

  uint4 kf[2][KG], vf[4][VG];
  auto load_k = [&](int tile) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int n = tile * 16 + r + 8 * i;
      const T* row = kb + n * p.k_sN;
#pragma unroll
      for (int g = 0; g < KG; ++g) kf[i][g] = ldg_stream(row + g * 32, n < p.n_keys && (DP == 128 || g * 32 + t * 8 < p.D));
    }
  };
  auto load_v = [&](int tile) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = tile * 16 + 2 * t + (i & 1) + 8 * (i >> 1);
      const T* row = vb + n * p.v_sN;
#pragma unroll
      for (int g = 0; g < VG; ++g) vf[i][g] = ldg_stream(row + g * 64, n < p.n_keys && (DP == 128 || r * 8 < p.D));
    }
  };
  float bf[NQ][4];
  auto load_b = [&](int tile) {
    if constexpr (BIAS != 0) {
#pragma unroll
      for (int n = 0; n < NQ; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int m = n * 8 + 2 * t + (i & 1), key = tile * 16 + r + 8 * (i >> 1);
          bf[n][i] = m < p.M && key < p.n_keys ? load_bias<BIAS, T>(p, bias_bh + m * p.bias_sM + key) : 0.f;
        }
    }
  };

  float o[NQ][VG * 4][4];  // O^T: [query group][16 head-dim rows][fragment]
#pragma unroll
  for (int n = 0; n < NQ; ++n)
#pragma unroll
    for (int i = 0; i < VG * 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[n][i][e] = 0.f;
  float mx[NQ][2], l[NQ][2];  // of queries 2t, 2t+1: running maximum (log2 units), this lane's part of the sum
#pragma unroll
  for (int n = 0; n < NQ; ++n) mx[n][0] = mx[n][1] = -INFINITY, l[n][0] = l[n][1] = 0.f;

  // The leaf in the accumulators is complete: into the warp's partial result `slot`, which it starts or follows.
  auto close_leaf = [&](int slot, bool starts) {
    float m_new[NQ][2];
#pragma unroll
    for (int n = 0; n < NQ; ++n)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int m = n * 8 + 2 * t + j, at = slot * p.M + m;
        m_new[n][j] = mx[n][j];
        if (m < p.M) {
          // lane (r, t) holds head-dim elements 64 g + 8 r .. + 7 of its query rows, and part r of their sums
          float* row = sm.o + at * Smem::kRow;
          float fa = 0.f, fx = 1.f;
          if (!starts) {
            const float m_old = sm.m[at];
            m_new[n][j] = fmaxf(m_old, mx[n][j]);
            fa = weight_of(m_old, m_new[n][j]);
            fx = weight_of(mx[n][j], m_new[n][j]);
            l[n][j] = fold2(fa, row[DP + r], fx, l[n][j]);
          }
          row[DP + r] = l[n][j];
#pragma unroll
          for (int i = 0; i < VG * 4; i += 2) {
            float4 v = make_float4(o[n][i][j], o[n][i][j + 2], o[n][i + 1][j], o[n][i + 1][j + 2]);
            float4& dst = *reinterpret_cast<float4*>(row + (i >> 2) * 64 + r * 8 + (i & 3) * 2);
            if (!starts) {
              const float4 a = dst;
              v = make_float4(fold2(fa, a.x, fx, v.x), fold2(fa, a.y, fx, v.y), fold2(fa, a.z, fx, v.z),
                              fold2(fa, a.w, fx, v.w));
            }
            dst = v;
          }
        }
        mx[n][j] = -INFINITY;
        l[n][j] = 0.f;
      }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (r == 0 && n * 8 + 2 * t + j < p.M) sm.m[slot * p.M + n * 8 + 2 * t + j] = m_new[n][j];
#pragma unroll
      for (int i = 0; i < VG * 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][i][e] = 0.f;
    }
    __syncwarp();
  };

  if (first < last) {
    load_k(first);
    load_b(first);
    load_v(first);
  }
  int left = p.leaf, leaf = 0;  // tiles left of the running leaf; leaves closed so far
#pragma unroll 1
  for (int tile = first; tile < last; ++tile) {
    float s[NQ][4];
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
      s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
      for (int g = 0; g < KG; ++g) {
        mma16816<T>(s[n], kf[0][g].x, kf[1][g].x, kf[0][g].y, kf[1][g].y, q[n][g].x, q[n][g].y);
        mma16816<T>(s[n], kf[0][g].z, kf[1][g].z, kf[0][g].w, kf[1][g].w, q[n][g].z, q[n][g].w);
      }
    }
    const bool more = tile + 1 < last;
    if (more) load_k(tile + 1);
    // scores in log2 units, -inf where masked
    bool need = false;
#pragma unroll
    for (int n = 0; n < NQ; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x = s[n][i] * p.sm_scale;
        // a mask selects: whatever the score of a masked key is (infinite, NaN), it takes no part
        if (BIAS == 2) x = bf[n][i] != 0.f ? x : -INFINITY;
        else if (BIAS != 0) x += bf[n][i];
        const int key = tile * 16 + r + 8 * (i >> 1);
        if (key >= p.n_keys || (p.causal && key > n * 8 + 2 * t + (i & 1))) x = -INFINITY;
        s[n][i] = x * kLog2e;
        need = need || s[n][i] > mx[n][i & 1] + 8.f;
      }
    if (more) load_b(tile + 1);
    if (__any_sync(0xffffffffu, need)) {
#pragma unroll
      for (int n = 0; n < NQ; ++n)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float m_new = fmaxf(mx[n][j], fmaxf(s[n][j], s[n][j + 2]));
          for (int off = 4; off < 32; off <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, off));
          const float alpha = m_new == -INFINITY ? 1.f : ex2(mx[n][j] - m_new);
          mx[n][j] = m_new;
          l[n][j] *= alpha;
#pragma unroll
          for (int i = 0; i < VG * 4; ++i) o[n][i][j] *= alpha, o[n][i][j + 2] *= alpha;
        }
    }
    uint32_t pb[NQ][2];
#pragma unroll
    for (int n = 0; n < NQ; ++n) {
      const float m0 = mx[n][0] == -INFINITY ? 0.f : mx[n][0], m1 = mx[n][1] == -INFINITY ? 0.f : mx[n][1];
      const float p0 = ex2(s[n][0] - m0), p1 = ex2(s[n][1] - m1), p2 = ex2(s[n][2] - m0), p3 = ex2(s[n][3] - m1);
      l[n][0] += p0 + p2;
      l[n][1] += p1 + p3;
      pb[n][0] = transpose8x8(P2::pack(p0, p1));
      pb[n][1] = transpose8x8(P2::pack(p2, p3));
    }
#pragma unroll
    for (int g = 0; g < VG; ++g) {
      const uint32_t w[4][4] = {{vf[0][g].x, vf[0][g].y, vf[0][g].z, vf[0][g].w},
                                {vf[1][g].x, vf[1][g].y, vf[1][g].z, vf[1][g].w},
                                {vf[2][g].x, vf[2][g].y, vf[2][g].z, vf[2][g].w},
                                {vf[3][g].x, vf[3][g].y, vf[3][g].z, vf[3][g].w}};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t a0 = __byte_perm(w[0][i], w[1][i], 0x5410), a1 = __byte_perm(w[0][i], w[1][i], 0x7632);
        const uint32_t a2 = __byte_perm(w[2][i], w[3][i], 0x5410), a3 = __byte_perm(w[2][i], w[3][i], 0x7632);
#pragma unroll
        for (int n = 0; n < NQ; ++n) mma16816<T>(o[n][g * 4 + i], a0, a1, a2, a3, pb[n][0], pb[n][1]);
      }
    }
    if (more) load_v(tile + 1);
    if (--left == 0 || !more) {
      close_leaf(warp * p.own + (p.fold == 1 ? leaf : leaf / kGroup), p.fold == 1 || leaf % kGroup == 0);
      ++leaf;
      left = p.leaf;
    }
  }

  __syncthreads();
  const int n_leaves = (n_tiles + p.leaf - 1) / p.leaf;
  const int n_groups = (n_leaves + kGroup - 1) / kGroup;
  const int cta_groups = W * p.own * p.fold / kGroup;
  if (p.fold == 1) {
    // ---- this CTA's leaves into groups, in the place of each group's first leaf
    const int here = min(n_leaves - static_cast<int>(blockIdx.x) * W * p.own, W * p.own);
    const int size = p.M * Smem::kRow;
    for (int e = tid; e < (here + kGroup - 1) / kGroup * size; e += W * 32) {
      const int g = e / size, at = e - g * size, m = at / Smem::kRow;
      const int s0 = g * kGroup;
      float acc = sm.o[s0 * size + at], m_acc = sm.m[s0 * p.M + m];
      for (int sx = s0 + 1; sx < min(here, s0 + kGroup); ++sx) {
        const float m_x = sm.m[sx * p.M + m], m_new = fmaxf(m_acc, m_x);
        acc = fold2(weight_of(m_acc, m_new), acc, weight_of(m_x, m_new), sm.o[sx * size + at]);
        m_acc = m_new;
      }
      sm.o[s0 * size + at] = acc;
      if (at == m * Smem::kRow) sm.gm[s0 * p.M + m] = m_acc;
    }
  }
  // ---- the head's result: each CTA finishes a share of the elements
  const int parts = static_cast<int>(gridDim.x);
  cg::cluster_group cluster = cg::this_cluster();
  if (parts > 1)
    cluster.sync();
  else
    __syncthreads();
  // a group: the CTA that has it, and its (first) place there
  const int rank = lane / cta_groups, place = lane % cta_groups * (kGroup / p.fold);
  auto of_group = [&](float* mine) -> float* { return parts > 1 ? cluster.map_shared_rank(mine, rank) : mine; };
  if (warp == 0 && lane < n_groups) sm.group[lane] = of_group(sm.o + place * p.M * Smem::kRow);
  for (int m = warp; live && m < p.M; m += W) {  // a warp per row, a lane per group
    float gm = -INFINITY, gl = 0.f;
    if (lane < n_groups) {
      gm = *of_group((p.fold == 1 ? sm.gm : sm.m) + place * p.M + m);
      const float4* part = reinterpret_cast<const float4*>(of_group(sm.o + (place * p.M + m) * Smem::kRow + DP));
      const float4 a = part[0], b4 = part[1];
      gl = ((a.x + a.y) + (a.z + a.w)) + ((b4.x + b4.y) + (b4.z + b4.w));
    }
    float m_all = gm;
    for (int off = 1; off < 32; off <<= 1) m_all = fmaxf(m_all, __shfl_xor_sync(0xffffffffu, m_all, off));
    const float f = weight_of(gm, m_all);
    float sum = __fmul_rn(f, gl);
    for (int off = 1; off < 32; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    sm.weight[m][lane] = f;
    if (lane == 0) sm.m_all[m] = m_all, sm.l_all[m] = sum;
  }
  __syncthreads();
  for (int e = static_cast<int>(blockIdx.x) * W * 32 + tid; live && e < p.M * DP; e += parts * W * 32) {
    const int m = e / DP, d = e - m * DP;
    float acc = 0.f;
#pragma unroll 8
    for (int g = 0; g < n_groups; ++g)
      acc = __fmaf_rn(sm.weight[m][g], sm.group[g][m * Smem::kRow + d], acc);
    // A row whose keys are all masked out: output 0, log-sum-exp +inf.  A NaN sum ends here too, and the product
    // with zero lets the NaN of its accumulators through (the tile kernel does the same).
    const float m_all = sm.m_all[m], sum = sm.l_all[m];
    const bool any_key = m_all != -INFINITY && sum > 0.f;
    if (d < p.D)
      (static_cast<T*>(p.o) + b * p.o_sB + m * p.o_sM + h * p.o_sH)[d] = static_cast<T>(any_key ? acc / sum : acc * 0.f);
    if (d == 0) p.lse[static_cast<int64_t>(bh) * p.M + m] = any_key ? m_all + log2f(sum) : INFINITY;
  }
  if (parts > 1) cluster.sync();  // no CTA leaves while another still reads its shared memory
}

// How many clusters of 1 .. 16 CTAs of a kernel the current device holds at once (asked once).
constexpr int kMaxParts = 16;
template <auto kern>  // one table per kernel
const int* resident_clusters(int warps, int smem) {
  static int table[64][kMaxParts + 1] = {};
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  int* t = table[dev];
  if (t[0] == 0) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return nullptr;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return nullptr;
    for (int parts = 1; parts <= kMaxParts; ++parts) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(parts, 1);
      cfg.blockDim = dim3(warps * 32);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = parts;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;  // this size is not launched
      }
      t[parts] = n;
    }
    t[0] = 1;
  }
  return t;
}

// Tiles in a leaf: a function of the number of keys and query rows alone.  Closing a leaf takes a quarter of a
// tile's instructions, more with many rows, so a leaf has a few tiles where there are enough; and there are no
// more leaves than the warps of a cluster can use - fewer for many rows, of which a warp can keep only two.
int leaf_tiles(int tiles, int rows) {
  const int most = rows <= 4 ? 120 : 64;
  static_assert(120 <= kMaxLeaves);
  const int least = tiles < 64 ? 2 : (rows <= 8 || tiles < 128 ? 4 : 8);
  return tiles <= least * most ? least : (tiles + most - 1) / most;
}

// The split of a (batch, head)'s leaves over the warps of `parts` CTAs: the one with the least
// (turns of the resident clusters) x (tiles per warp + the start and the merge of a CTA, which take
// about as long as six tiles).  A single turn that fills the SMs wins where there are few heads,
// several turns of longer CTAs where there are many.  (With a split free of leaves, and so results that depend on the
// number of heads: B8 H32 N4096 90 us, B1 H32 N20011 61, B64 H32 N2048 319, B32 H32 N1000 D64 50.)
struct Split {
  int parts = 0, warps = 0, fold = 0, own = 0;
  int64_t cost = -1;
};
void consider(Split& best, const int* resident, int warps, int slots, int bh, int tiles, int leaf) {
  if (!resident) return;
  const int leaves = (tiles + leaf - 1) / leaf;
  for (int fold = 1; fold <= kGroup; fold += kGroup - 1)
    for (int own = 1; own <= slots; ++own) {
      const int parts = (leaves + warps * own * fold - 1) / (warps * own * fold);
      if (parts > kMaxParts || resident[parts] < 1) continue;
      const int64_t turns = (bh + resident[parts] - 1) / resident[parts];
      const int per_warp = own * fold * leaf;
      const int64_t cost = turns * ((per_warp < tiles ? per_warp : tiles) + 6);
      if (best.cost < 0 || cost < best.cost) best = {parts, warps, fold, own, cost};
    }
}

template <int DP, int NQ, typename T, int BIAS>
int launch_inst(DecodeParams dp, int bh, cudaStream_t stream) {
  const int tiles = (dp.n_keys + 15) / 16;
  dp.leaf = leaf_tiles(tiles, dp.M);
  constexpr int kSmem4 = sizeof(DecodeSmem<DP, NQ, 4>);
  Split s;
  consider(s, resident_clusters<decode_kernel<DP, NQ, 4, T, BIAS>>(4, kSmem4), 4, DecodeSmem<DP, NQ, 4>::slots(dp.M), bh, tiles, dp.leaf);
  // twice the warps per head where even 16 CTAs leave SMs idle (one group of rows only: with two the
  // registers do not allow it)
  constexpr int kSmem8 = sizeof(DecodeSmem<DP, 1, 8>);
  if constexpr (NQ == 1)
    consider(s, resident_clusters<decode_kernel<DP, NQ, 8, T, BIAS>>(8, kSmem8), 8, DecodeSmem<DP, NQ, 8>::slots(dp.M), bh, tiles, dp.leaf);
  if (s.cost < 0) return FA_ERR_CUDA;
  dp.fold = s.fold;
  dp.own = s.own;
  if constexpr (NQ == 1)
    if (s.warps == 8)
      return launch_overlapped(decode_kernel<DP, NQ, 8, T, BIAS>, dim3(s.parts, bh), 256, kSmem8, stream, dp, s.parts);
  return launch_overlapped(decode_kernel<DP, NQ, 4, T, BIAS>, dim3(s.parts, bh), 128, kSmem4, stream, dp, s.parts);
}

template <int DP, typename T, int BIAS>
int launch_rows(const DecodeParams& dp, int bh, cudaStream_t stream) {
  return dp.M <= 8 ? launch_inst<DP, 1, T, BIAS>(dp, bh, stream) : launch_inst<DP, 2, T, BIAS>(dp, bh, stream);
}

template <int DP, typename T>
int launch_bias(const DecodeParams& dp, int bias_kind, int bh, cudaStream_t stream) {
  switch (bias_kind) {
    case FA_BIAS_NONE: return launch_rows<DP, T, 0>(dp, bh, stream);
    case FA_BIAS_SAME: return launch_rows<DP, T, 1>(dp, bh, stream);
    case FA_BIAS_BOOL: return launch_rows<DP, T, 2>(dp, bh, stream);
    case FA_BIAS_F32: return launch_rows<DP, T, 3>(dp, bh, stream);
    default: return FA_ERR_UNSUPPORTED;
  }
}

template <typename T>
int launch_dtype(const DecodeParams& dp, int bias_kind, int bh, cudaStream_t stream) {
  return dp.D <= 64 ? launch_bias<64, T>(dp, bias_kind, bh, stream)
                    : launch_bias<128, T>(dp, bias_kind, bh, stream);
}

}  // namespace

// 16 rows are what two groups of 8 queries cover; at head dim 256 the operands no longer fit a
// thread's registers.
bool decode_takes(int M, int D) { return M <= 16 && D <= 128; }

int launch_decode(const fa_params& p, cudaStream_t stream, int* status) {
  auto bad = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 16 != 0 || s[0] % 8 || s[1] % 8 || s[2] % 8;
  };
  if (!operand_ok(p.q, p.q_stride) || !operand_ok(p.k, p.k_stride) || !operand_ok(p.v, p.v_stride) || bad(p.o, p.o_stride))
    return FA_ERR_ALIGN;
  DecodeParams d;
  d.q = p.q;
  d.k = p.k;
  d.v = p.v;
  d.bias = p.bias;
  d.o = p.o;
  d.lse = p.lse;
  d.status = status;
  d.q_sB = p.q_stride[0], d.q_sM = p.q_stride[1], d.q_sH = p.q_stride[2];
  d.k_sB = p.k_stride[0], d.k_sN = p.k_stride[1], d.k_sH = p.k_stride[2];
  d.v_sB = p.v_stride[0], d.v_sN = p.v_stride[1], d.v_sH = p.v_stride[2];
  d.o_sB = p.o_stride[0], d.o_sM = p.o_stride[1], d.o_sH = p.o_stride[2];
  d.bias_sB = p.bias_stride[0], d.bias_sH = p.bias_stride[1], d.bias_sM = p.bias_stride[2];
  d.H = p.H, d.M = p.M, d.N = p.N, d.D = p.D;
  d.n_keys = p.causal && p.M < p.N ? p.M : p.N;
  d.causal = p.causal ? 1 : 0;
  d.sm_scale = p.sm_scale;
  const int bh = p.B * p.H;
  return p.dtype == FA_BF16 ? launch_dtype<__nv_bfloat16>(d, p.bias_kind, bh, stream)
                            : launch_dtype<__half>(d, p.bias_kind, bh, stream);
}

}  // namespace fa
