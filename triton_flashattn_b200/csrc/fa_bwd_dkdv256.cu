// dV (and dS) kernel for head dimension 256 on sm_100a; dK follows as a streamed product.
//
// At D = 256 the accumulators dV and dK of 128 keys alone fill the 512 tensor-memory columns, and
// the tiles of K, V, Q, dO of a [128 x 128] step would take 256 KB.  The 16-bit dS has to go out to
// global memory anyway (dQ = sm_scale * dS K is a streamed product at this head dimension), so dK
// is one too:
//   this kernel     S = Q K^T, dP = dO V^T, P, dS -> global, dV += P^T dO   (S | dP | dV: 512 columns)
//   fa_bwd_dq.cu    dK = sm_scale * dS^T Q, then dQ = sm_scale * dS K
// Persistent, one CTA per SM.  A tile is 128 keys of one (batch, head); a CTA walks its tiles and,
// inside a tile, the 128-row query blocks that see its keys.  K and V stay in shared memory for a
// tile (64 KB each); Q and dO pass through a ring of two 32 KB stages, each [128 rows][128 head-dim
// columns], in the order the products take them:
//   Q(0) | Q(1) dO(0) | Q(2) dO(1) | ...
// so S of the next step is computed while the row threads form P of this one.  The last 32 KB are P;
// a 16-bit bias tile lands there by TMA first, each thread reads the chunks it overwrites with P.
// Roles (640 threads):
//   warps 0-15  row threads: tensor-memory lanes 32*(w&3).. (query rows), 32-key column quarter w>>2
//   warps 16/17 TMA producers: each brings one of the two 16 KB boxes of every stage and half of K
//               and V (one thread's stream of boxes reaches 24 bytes per cycle, a step needs 30)
//   warp 18     MMA issuer, tensor-memory owner
//   warp 19     TMA loads of the 16-bit bias tiles
// The control warps walk their loops converged and elect a lane for the issue.
// Rule kept by every barrier here: the next completion of a barrier needs progress of every thread
// that waits on it, so a parity wait can never be two phases behind.
//
// What bounds it: a step is 128 KB of Q / dO against 3072 cycles of products, with one ring turn
// (product, hand-back, load) exposed per step.  The version before kept dV^T and dK^T of 64 keys in
// one kernel with everything single-staged: 11,900 cycles a step of half the keys.
// B4 H8 S2048, 16-bit bias: 0.33 ms and 0.075 ms for dK; the training pass 957 -> 731 us.
//
// Query blocks above the causal diagonal are not visited: the caller zero-fills dbias.
//
// Replaces _attn_bwd_dkdv / _attn_bwd_dkdv_inner of the reference (flash_attention.py
// 237-454) at BLOCK_HEADDIM = 256: same P, dS, dbias = dS, dK scaled by sm_scale.
#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

struct Dkdv256Params {
  CUtensorMap map_q;   // boxes of 128 rows
  CUtensorMap map_k;
  CUtensorMap map_v;
  CUtensorMap map_do;
  CUtensorMap map_bias;
  const void* bias;
  void* dv;
  void* ds16;        // (B, H, M, N) 16-bit dS out; rows 16-byte aligned
  float* dbias_f32;  // fp32 bias gradient or null
  const float* lse;
  const float* delta;
  int* status;
  int64_t bias_sB, bias_sH, bias_sM;
  int64_t ds_sB, ds_sH, ds_sM;
  int64_t dbf_sB, dbf_sH, dbf_sM;
  int64_t dv_sB, dv_sN, dv_sH;
  int H, M, N;
  int n_nblk, n_tiles;  // key blocks per (batch, head); tiles of this launch
  int bh0;              // first (batch, head) of this launch
  int ds_flat;          // ds16 holds slabs numbered from bh0 (ds_sH apart) instead of a (B, H, M, N) tensor
  int causal, bias_vec32, bias_b_mul, bias_h_mul;
  int ds_vec32, dv_vec32;  // bases and strides are multiples of 32 bytes
  float scale_log2;        // sm_scale * log2(e)
};

enum Dkdv256Site { kSiteKFull = 1, kSiteKEmpty, kSiteVFull, kSiteVEmpty, kSiteFull, kSiteEmpty, kSiteSFull,
                   kSiteSFree, kSitePReady, kSiteDpFull, kSiteDvDone, kSiteBiasFull, kSiteEpilogue };

constexpr int kTile256 = 128 * 256 * 2;  // K or V: four [128][64] blocks
constexpr int kStage256 = 2 * kBlk;      // [128 rows][128 columns] of Q or dO
constexpr int kOffK = 0, kOffV = kOffK + kTile256, kOffRing = kOffV + kTile256;
constexpr int kOffP = kOffRing + 2 * kStage256;
constexpr int kSmem256 = kOffP + 2 * kBlk + 1024;  // + slack for 1024-byte alignment

// 32 bytes: one sector store, or two halves where the address is only 16-byte aligned
__device__ __forceinline__ void store32(void* dst, const uint32_t* w, bool vec32) {
  if (vec32) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

template <typename T, int BIAS>
__global__ void __launch_bounds__(640, 1) dkdv256_kernel(const __grid_constant__ Dkdv256Params p) {
  using P2 = Pack2<T>;
  constexpr uint32_t kColS = 0, kColDp = 128, kColDv = 256;
  constexpr uint32_t kTmemCols = 512;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t k_full, k_empty, v_full, v_empty, full[2], empty[2];
  __shared__ uint64_t s_full, s_free, p_ready, dp_full, dv_done, bias_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int tid = threadIdx.x;
  // the warp index as a value the compiler knows to be the same in all lanes
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int n_mblk = (p.M + 127) >> 7;

  // Tiles as in the dK/dV kernel of the smaller head dims: (batch*head)-major, CTA c takes units
  // c, c+G, ...; a causal unit is a heavy and a light key block.
  const int sched_sh = p.causal ? 1 : 0;
  auto tile_at = [&](int it, int& bh, int& nb, int& i_start) -> bool {
    const int u = static_cast<int>(blockIdx.x) + (it >> sched_sh) * static_cast<int>(gridDim.x);
    const int k = (u << sched_sh) + (it & sched_sh);
    if (k >= p.n_tiles) return false;
    bh = k / p.n_nblk;
    const int pos = k - bh * p.n_nblk;
    bh += p.bh0;
    nb = p.causal ? ((pos & 1) ? p.n_nblk - 1 - (pos >> 1) : (pos >> 1)) : pos;
    // causal (top-left aligned): query block i sees key block nb when i >= nb
    i_start = p.causal ? min(nb, n_mblk) : 0;
    return true;
  };
  // Walks the steps (tile, query block) of this CTA.
  struct Step {
    int it = -1, bh = 0, nb = 0, mb = 0;
    bool first = false, valid = true;  // first step of its tile
  };
  auto next_step = [&](Step& s) {
    if (s.it >= 0 && s.mb + 1 < n_mblk) {
      ++s.mb;
      s.first = false;
      return;
    }
    do {
      ++s.it;
      s.valid = tile_at(s.it, s.bh, s.nb, s.mb);
    } while (s.valid && s.mb >= n_mblk);  // tiles no query row sees have no step
    s.first = true;
  };

  WaitCtx ctx{&abort_flag, p.status, 5};

  if (tid == 0) {
    abort_flag = 0;
    mbar_init(&k_full, 2);
    mbar_init(&k_empty, 1);
    mbar_init(&v_full, 2);
    mbar_init(&v_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], 2);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&s_free, 16);
    mbar_init(&p_ready, 16);
    mbar_init(&dp_full, 1);
    mbar_init(&dv_done, 1);
    mbar_init(&bias_full, 1);
    mbar_fence_init();
  }
  if (warp == 18) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  grid_dep_launch_next();
  grid_dep_wait();  // the previous kernels' results (and the status word) are visible from here
  const bool live = *reinterpret_cast<volatile int*>(p.status) == 0;

  if (warp == 16 || warp == 17) {
    // ----------------------------------------------------------------- producers
    if (live) {
      const int half = warp - 16;
      if (lane == 0) {
        tma_prefetch_desc(&p.map_q);
        tma_prefetch_desc(&p.map_k);
        tma_prefetch_desc(&p.map_v);
        tma_prefetch_desc(&p.map_do);
      }
      bool ok = true;
      uint32_t use = 0;          // ring stages filled so far
      uint32_t nk = 0, nv = 0;   // K / V tiles asked for so far
      // this producer's two blocks (64 columns each) of a K or V tile
      auto tile_load = [&](const CUtensorMap* map, int off, uint64_t* bar, const Step& s) {
        const int b = s.bh / p.H, h = s.bh - b * p.H;
        if (elect_one()) {
          mbar_expect_tx(bar, kTile256 / 2);
          for (int kb = 2 * half; kb < 2 * half + 2; ++kb)
            tma_load_4d(smem + off + kb * kBlk, map, bar, kb * 64, h, s.nb * 128, b);
        }
        __syncwarp();
      };
      // both column halves of a query block of Q or dO, a stage each
      auto ring_load = [&](const CUtensorMap* map, const Step& s) -> bool {
        const int b = s.bh / p.H, h = s.bh - b * p.H;
        for (int c = 0; c < 2; ++c, ++use) {
          const uint32_t st = use & 1;
          if (use >= 2 && !wait_warp(&empty[st], ((use >> 1) - 1) & 1, ctx, kSiteEmpty, s.mb)) return false;
          if (elect_one()) {
            mbar_expect_tx(&full[st], kBlk);
            tma_load_4d(smem + kOffRing + st * kStage256 + half * kBlk, map, &full[st], c * 128 + half * 64, h,
                        s.mb * 128, b);
          }
          __syncwarp();
        }
        return true;
      };
      Step cur, prev;
      prev.valid = false;
      next_step(cur);
      while (ok && (cur.valid || prev.valid)) {
        if (cur.valid) {
          if (cur.first) {
            if (nk >= 1) ok = wait_warp(&k_empty, (nk - 1) & 1, ctx, kSiteKEmpty, cur.it);
            if (!ok) break;
            ++nk;
            tile_load(&p.map_k, kOffK, &k_full, cur);
          }
          if (BIAS != 0 && half == 0) {
            // the bias tile of this step is pulled into L2, about a step before it is read
            constexpr int kBox = BIAS == 1 ? 64 : (BIAS == 3 ? 32 : 128);  // keys per box of map_bias
            const int b = cur.bh / p.H, h = cur.bh - b * p.H;
            if (elect_one()) {
#pragma unroll
              for (int c = 0; c < 128; c += kBox)
                if (cur.nb * 128 + c < p.N)
                  tma_prefetch_l2_4d(&p.map_bias, cur.nb * 128 + c, cur.mb * 128, h * p.bias_h_mul, b * p.bias_b_mul);
            }
            __syncwarp();
          }
          ok = ring_load(&p.map_q, cur);
          if (!ok) break;
        }
        if (prev.valid) {
          if (prev.first) {
            if (nv >= 1) ok = wait_warp(&v_empty, (nv - 1) & 1, ctx, kSiteVEmpty, prev.it);
            if (!ok) break;
            ++nv;
            tile_load(&p.map_v, kOffV, &v_full, prev);
          }
          ok = ring_load(&p.map_do, prev);
        }
        prev = cur;
        if (cur.valid) next_step(cur);
      }
    }
  } else if (warp == 18) {
    // --------------------------------------------------------------- MMA issuer
    if (live) {
      constexpr bool bf = P2::kIsBf16;
      constexpr uint32_t idesc_s = make_idesc(bf, false, false, 128, 128);
      constexpr uint32_t idesc_g = make_idesc(bf, true, true, 128, 128);
      const uint64_t k_km = make_sdesc(smem_u32(smem + kOffK), 0, 1024), v_km = make_sdesc(smem_u32(smem + kOffV), 0, 1024);
      const uint64_t p_mn = make_sdesc(smem_u32(smem + kOffP), kBlk, 1024);
      const uint32_t ring = smem_u32(smem + kOffRing);
      constexpr uint64_t kHalfTile = static_cast<uint64_t>(2 * kBlk) >> 4;  // two blocks, in descriptor units
      bool ok = true;
      uint32_t use = 0;         // ring stages taken so far
      uint32_t nk = 0, nv = 0;  // K / V tiles taken so far
      uint32_t g = 0;           // steps whose S was issued
      Step cur, prev;
      prev.valid = false;
      next_step(cur);
      while (ok && (cur.valid || prev.valid)) {
        const Step here = cur;
        if (cur.valid) next_step(cur);
        if (here.valid) {
          // S of step g: its columns are free once the row threads hold S of step g-1
          if (here.first) {
            ok = wait_warp(&k_full, nk & 1, ctx, kSiteKFull, here.it);
            ++nk;
          }
          if (ok && g >= 1) ok = wait_warp_hot(&s_free, (g - 1) & 1, ctx, kSiteSFree, here.mb);
          for (int c = 0; c < 2 && ok; ++c, ++use) {
            const uint32_t st = use & 1;
            ok = wait_warp_hot(&full[st], (use >> 1) & 1, ctx, kSiteFull, here.mb);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
              issue_gemm_ss<8, false, false>(tmem + kColS, make_sdesc(ring + st * kStage256, 0, 1024),
                                             k_km + c * kHalfTile, kBlk, kBlk, idesc_s, c > 0);
              mma_commit(&empty[st]);
              if (c == 1) {
                mma_commit(&s_full);
                if (cur.valid && cur.first) mma_commit(&k_empty);  // last step of its tile: K may be replaced
              }
            }
            __syncwarp();
          }
          if (!ok) break;
          ++g;
        }
        if (prev.valid) {
          // dP and dV of the step before.  All sixteen row warps announce P after they have read dP of
          // the step before that and, at the start of a tile, the finished dV of the last one.
          const uint32_t gp = here.valid ? g - 2 : g - 1;
          if (prev.first) {
            ok = wait_warp(&v_full, nv & 1, ctx, kSiteVFull, prev.it);
            ++nv;
          }
          if (ok) ok = wait_warp_hot(&p_ready, gp & 1, ctx, kSitePReady, prev.mb);
          for (int c = 0; c < 2 && ok; ++c) {
            const uint32_t st = (use + c) & 1;
            ok = wait_warp_hot(&full[st], ((use + c) >> 1) & 1, ctx, kSiteFull, prev.mb);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
              issue_gemm_ss<8, false, false>(tmem + kColDp, make_sdesc(ring + st * kStage256, 0, 1024),
                                             v_km + c * kHalfTile, kBlk, kBlk, idesc_s, c > 0);
              if (c == 1) {
                mma_commit(&dp_full);
                if (!here.valid || here.first) mma_commit(&v_empty);  // last step of its tile
              }
            }
            __syncwarp();
          }
          if (!ok) break;
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              const uint32_t st = (use + c) & 1;
              issue_gemm_ss<8, true, true>(tmem + kColDv + c * 128, p_mn, make_sdesc(ring + st * kStage256, kBlk, 1024),
                                           kBlk, kBlk, idesc_g, !prev.first);
              mma_commit(&empty[st]);
            }
            mma_commit(&dv_done);
          }
          __syncwarp();
          use += 2;
        }
        prev = here;
      }
    }
    __syncwarp();
  } else if (warp == 19) {
    // ----------------------------------------------------------- bias tile loads
    if (BIAS == 1 && live) {
      if (lane == 0) tma_prefetch_desc(&p.map_bias);
      bool ok = true;
      Step s;
      next_step(s);
      for (uint32_t gs = 0; s.valid; ++gs, next_step(s)) {
        // the P tile is free once dV of the previous step has read it
        if (gs >= 1) ok = wait_warp_hot(&dv_done, (gs - 1) & 1, ctx, kSiteDvDone, s.mb);
        if (!ok) break;
        const int b = s.bh / p.H, h = s.bh - b * p.H, n0 = s.nb * 128;
        const bool two = n0 + 64 < p.N;
        if (elect_one()) {
          mbar_expect_tx(&bias_full, two ? 2 * kBlk : kBlk);
          tma_load_4d(smem + kOffP, &p.map_bias, &bias_full, n0, s.mb * 128, h * p.bias_h_mul, b * p.bias_b_mul);
          if (two)
            tma_load_4d(smem + kOffP + kBlk, &p.map_bias, &bias_full, n0 + 64, s.mb * 128, h * p.bias_h_mul,
                        b * p.bias_b_mul);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    // --------------------------------------------------------------- row threads
    const int r = (warp & 3) * 32 + lane;  // query row inside the block = tensor-memory lane
    const int qt = warp >> 2;              // column quarter: keys n0 + 32*qt .. +31
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    bool ok = live;
    // this thread's four 16-byte chunks of P: chunk c at sp_row + ((chunk0 + c) ^ (r & 7)) * 16
    const uint32_t sp_row = smem_u32(smem + kOffP + (qt >> 1) * kBlk) + static_cast<uint32_t>(r) * 128u;
    const uint32_t chunk0 = (qt & 1) * 4;
    const uint32_t tm_sc = tmem_addr(tmem, lane_base, kColS + qt * 32);

    constexpr int BR = BIAS == 2 ? 2 : 0;  // the byte mask is read one step ahead
    BiasRegs<BR> bnext;
    // -LSE2 and delta of the coming step's row, as loaded: looked at when that step starts
    float lse_next = 0.f, delta_next = 0.f;
    auto prefetch = [&](int bh_, int c0, int mblk) {
      const int m = mblk * 128 + r;
      if constexpr (BR == 2) {
        const int b_ = bh_ / p.H, h_ = bh_ - b_ * p.H;
        load_bias_row<2>(bnext, p.bias, b_ * p.bias_sB + h_ * p.bias_sH + (int64_t)m * p.bias_sM, m < p.M, c0, p.N,
                         p.bias_vec32 != 0);
      }
      const int64_t idx = (int64_t)bh_ * p.M + min(m, p.M - 1);
      lse_next = __ldcg(p.lse + idx);
      delta_next = __ldcg(p.delta + idx);
    };
    uint32_t gs = 0;  // steps done so far, over all tiles
    int bh, nb, i_start;
    if (ok && tile_at(0, bh, nb, i_start) && i_start < n_mblk) prefetch(bh, nb * 128 + qt * 32, i_start);
#pragma unroll 1
    for (int it = 0; ok && tile_at(it, bh, nb, i_start); ++it) {
      const int col0 = nb * 128 + qt * 32;
      const int b = bh / p.H, h = bh - b * p.H;
      const int64_t ds_bh = p.ds_flat ? (bh - p.bh0) * p.ds_sH : b * p.ds_sB + h * p.ds_sH;
#pragma unroll 1
      for (int mb = i_start; mb < n_mblk && ok; ++mb, ++gs) {
        const int m0 = mb * 128;
        const bool row_ok = m0 + r < p.M;
        BiasRegs<BR> bcur = bnext;
        BiasRegs<BIAS == 3 ? 3 : 0> bf32;
        // fp32 bias row of this step: asked for now, used once S has arrived
        if constexpr (BIAS == 3)
          load_bias_row<3>(bf32, p.bias, b * p.bias_sB + h * p.bias_sH + (int64_t)(m0 + r) * p.bias_sM, row_ok, col0, p.N,
                           p.bias_vec32 != 0);
        // rows beyond M get -inf / 0, which makes their P and dS zero
        const float neg_lse = row_ok ? -lse_next : -INFINITY, delta_r = row_ok ? delta_next : 0.f;
        if (mb + 1 < n_mblk) prefetch(bh, col0, mb + 1);

        // ---- P
        ok = wait_warp(&s_full, gs & 1, ctx, kSiteSFull, mb);
        if (!ok) break;
        tc_fence_after();
        float pr[32];
        tmem_ld32(tm_sc, reinterpret_cast<uint32_t*>(pr));
        tmem_ld_wait();
        // S now lives in registers: hand its columns back for the next S
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free);
        // P = exp2(S * scale * log2e + bias * log2e - LSE2)
        if constexpr (BIAS == 1) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const f32x2 x = ffma2(f2(pr[i], pr[i + 1]), f2(p.scale_log2, p.scale_log2), f2(neg_lse, neg_lse));
            pr[i] = f2_lo(x);
            pr[i + 1] = f2_hi(x);
          }
          ok = wait_warp(&bias_full, gs & 1, ctx, kSiteBiasFull, mb);
          if (!ok) break;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = lds128(sp_row + (((chunk0 + c) ^ (r & 7)) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = P2::unpack(w[e]);
              const int i = c * 8 + e * 2;
              const f32x2 a = ffma2(f2(f.x, f.y), f2(kLog2e, kLog2e), f2(pr[i], pr[i + 1]));
              pr[i] = ex2(f2_lo(a));
              pr[i + 1] = ex2(f2_hi(a));
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            f32x2 a = ffma2(f2(pr[i], pr[i + 1]), f2(p.scale_log2, p.scale_log2), f2(neg_lse, neg_lse));
            if constexpr (BIAS == 3)
              a = ffma2(f2(__uint_as_float(bf32.w[i]), __uint_as_float(bf32.w[i + 1])), f2(kLog2e, kLog2e), a);
            float e0 = ex2(f2_lo(a)), e1 = ex2(f2_hi(a));
            if constexpr (BIAS == 2) {
              const uint32_t m2 = bcur.w[i >> 2] >> (8 * (i & 3));
              e0 = (m2 & 0xFFu) != 0 ? e0 : 0.f;
              e1 = (m2 & 0xFF00u) != 0 ? e1 : 0.f;
            }
            pr[i] = e0;
            pr[i + 1] = e1;
          }
        }
        if ((col0 + 32 > p.N) || (p.causal && col0 + 31 > m0)) {
          int limit = p.N - col0;
          if (p.causal) limit = min(limit, m0 + r - col0 + 1);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i >= limit) pr[i] = 0.f;
        }
        // dV of the previous step has read P (the first step of a tile: seen in the epilogue)
        if (mb > i_start) {
          ok = wait_warp(&dv_done, (gs - 1) & 1, ctx, kSiteDvDone, mb);
          if (!ok) break;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
          sts128(sp_row + (((chunk0 + c) ^ (r & 7)) << 4), P2::pack(pr[c * 8 + 0], pr[c * 8 + 1]),
                 P2::pack(pr[c * 8 + 2], pr[c * 8 + 3]), P2::pack(pr[c * 8 + 4], pr[c * 8 + 5]),
                 P2::pack(pr[c * 8 + 6], pr[c * 8 + 7]));
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready);

        // ---- dS = P * (dP - delta)
        ok = wait_warp(&dp_full, gs & 1, ctx, kSiteDpFull, mb);
        if (!ok) break;
        tc_fence_after();
        T* drow = reinterpret_cast<T*>(p.ds16) + ds_bh + (int64_t)(m0 + r) * p.ds_sM + col0;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t dp[16];
          tmem_ld16(tm_sc + (kColDp - kColS) + hf * 16, dp);
          tmem_ld_wait();
          if (hf == 1) tc_fence_before();  // the next arrival on p_ready hands the dP columns back
          uint32_t dsu[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = hf * 16 + 2 * i;
            const f32x2 d = fmul2(f2(pr[e], pr[e + 1]),
                                  fadd2(f2(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])),
                                        f2(-delta_r, -delta_r)));
            dsu[i] = P2::pack(f2_lo(d), f2_hi(d));
            if (BIAS == 3) {
              dp[2 * i] = __float_as_uint(f2_lo(d));
              dp[2 * i + 1] = __float_as_uint(f2_hi(d));
            }
          }
          const int c0 = col0 + hf * 16;
          if (row_ok && c0 < p.N) {
            if (c0 + 16 <= p.N) {
              store32(drow + hf * 16, dsu, p.ds_vec32 != 0);
            } else {
              const uint16_t* e16 = reinterpret_cast<const uint16_t*>(dsu);
#pragma unroll
              for (int k = 0; k < 16; ++k)
                if (c0 + k < p.N) reinterpret_cast<uint16_t*>(drow)[hf * 16 + k] = e16[k];
            }
            if (BIAS == 3 && p.dbias_f32 != nullptr) {
              // the fp32 bias gradient goes out unrounded
              float* frow = p.dbias_f32 + b * p.dbf_sB + h * p.dbf_sH + (int64_t)(m0 + r) * p.dbf_sM + c0;
              if (c0 + 16 <= p.N) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  *reinterpret_cast<uint4*>(frow + 4 * k) = make_uint4(dp[4 * k], dp[4 * k + 1], dp[4 * k + 2], dp[4 * k + 3]);
              } else {
#pragma unroll
                for (int k = 0; k < 16; ++k)
                  if (c0 + k < p.N) frow[k] = __uint_as_float(dp[k]);
              }
            }
          }
        }
      }
      if (!ok) break;

      // the next tile's first rows travel while this tile's result is stored
      {
        int bh2, nb2, is2;
        if (tile_at(it + 1, bh2, nb2, is2) && is2 < n_mblk) prefetch(bh2, nb2 * 128 + qt * 32, is2);
      }

      // ---- epilogue: dV (rows = keys) -> global, 64 head-dim columns per thread
      const bool any = i_start < n_mblk;
      if (any) {
        ok = wait_warp(&dv_done, (gs - 1) & 1, ctx, kSiteEpilogue, 0);
        if (!ok) break;
      }
      tc_fence_after();
      const int n = nb * 128 + r;
      T* row = reinterpret_cast<T*>(p.dv) + b * p.dv_sB + (int64_t)n * p.dv_sN + h * p.dv_sH + qt * 64;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t a[32];
        if (any) {
          tmem_ld32(tm_sc - qt * 32 + kColDv + qt * 64 + hf * 32, a);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) a[i] = 0;  // keys no query row sees
        }
        if (n < p.N) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint4 lo = pack8<P2>(a + c * 16, 1.f), hi = pack8<P2>(a + c * 16 + 8, 1.f);
            const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            store32(row + hf * 32 + c * 16, w, p.dv_vec32 != 0);
          }
        }
      }
      // the accumulators are in registers: the next tile's first products may overwrite them
      tc_fence_before();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 18) tmem_dealloc(tmem, kTmemCols);
}

template <typename T, int BIAS>
int launch_inst(const Dkdv256Params& kp, dim3 grid, cudaStream_t stream) {
  auto kern = dkdv256_kernel<T, BIAS>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem256) != cudaSuccess)
      return FA_ERR_CUDA;
    configured[dev] = true;
  }
  return launch_overlapped(kern, grid, 640, kSmem256, stream, kp);
}

template <typename T>
int launch_bias(const Dkdv256Params& kp, int bias_kind, dim3 grid, cudaStream_t stream) {
  switch (bias_kind) {
    case FA_BIAS_NONE: return launch_inst<T, 0>(kp, grid, stream);
    case FA_BIAS_SAME: return launch_inst<T, 1>(kp, grid, stream);
    case FA_BIAS_BOOL: return launch_inst<T, 2>(kp, grid, stream);
    case FA_BIAS_F32: return launch_inst<T, 3>(kp, grid, stream);
    default: return FA_ERR_UNSUPPORTED;
  }
}

}  // namespace

// The 16-bit dS tensor of a head-dim-256 backward: the bias gradient itself when one is
// wanted for a 16-bit bias, otherwise the caller's scratch.
const void* d256_ds_tensor(const fa_params& p, const int64_t** stride) {
  if (p.write_dbias && p.bias_kind == FA_BIAS_SAME) {
    *stride = p.dbias_stride;
    return p.dbias;
  }
  *stride = p.ds16_stride;
  return p.ds16;
}

int launch_bwd_dkdv_d256(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab) {
  Dkdv256Params kp;
  int r = make_tmap_bshd(&kp.map_q, p.q, p.B, p.M, p.H, p.D, p.q_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_k, p.k, p.B, p.N, p.H, p.D, p.k_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_v, p.v, p.B, p.N, p.H, p.D, p.v_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_do, p.d_o, p.B, p.M, p.H, p.D, p.do_stride, 128);
  if (r) return r;
  const int64_t slab_stride[3] = {0, slab ? slab->pitch * p.M : 0, slab ? slab->pitch : 0};
  const int64_t* ds_stride = slab_stride;
  const void* ds = slab ? slab->base : d256_ds_tensor(p, &ds_stride);
  kp.bh0 = slab ? slab->bh0 : 0;
  kp.ds_flat = slab != nullptr;
  if (!ds) return FA_ERR_NULL;
  if (reinterpret_cast<uintptr_t>(ds) % 16 != 0 || ds_stride[0] % 8 || ds_stride[1] % 8 || ds_stride[2] % 8)
    return FA_ERR_ALIGN;
  kp.ds16 = const_cast<void*>(ds);
  kp.ds_sB = ds_stride[0];
  kp.ds_sH = ds_stride[1];
  kp.ds_sM = ds_stride[2];
  const bool f32 = p.bias_kind == FA_BIAS_F32;
  kp.dbias_f32 = nullptr;
  kp.dbf_sB = kp.dbf_sH = kp.dbf_sM = 0;
  if (f32 && p.write_dbias) {
    if (reinterpret_cast<uintptr_t>(p.dbias) % 16 != 0 || p.dbias_stride[0] % 4 || p.dbias_stride[1] % 4 ||
        p.dbias_stride[2] % 4)
      return FA_ERR_ALIGN;
    kp.dbias_f32 = static_cast<float*>(p.dbias);
    kp.dbf_sB = p.dbias_stride[0];
    kp.dbf_sH = p.dbias_stride[1];
    kp.dbf_sM = p.dbias_stride[2];
  }
  auto bad = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 16 != 0 || s[0] % 8 || s[1] % 8 || s[2] % 8;
  };
  if (bad(p.dk, p.dk_stride) || bad(p.dv, p.dv_stride)) return FA_ERR_ALIGN;
  const int eb = p.bias_kind == FA_BIAS_BOOL ? 1 : (f32 ? 4 : 2);
  if (p.bias_kind != FA_BIAS_NONE) {
    if (reinterpret_cast<uintptr_t>(p.bias) % 16 != 0 || (p.bias_stride[0] * eb) % 16 ||
        (p.bias_stride[1] * eb) % 16 || (p.bias_stride[2] * eb) % 16)
      return FA_ERR_ALIGN;
  }
  kp.bias_b_mul = kp.bias_h_mul = 0;
  kp.map_bias = kp.map_q;
  if (p.bias_kind != FA_BIAS_NONE) {
    const int box = p.bias_kind == FA_BIAS_SAME ? 64 : (f32 ? 32 : 128);
    r = make_tmap_bhmn(&kp.map_bias, p.bias, eb, p.B, p.H, p.M, p.N, p.bias_stride, box, 128, &kp.bias_b_mul,
                       &kp.bias_h_mul);
    if (r) return r;
  }
  kp.bias_vec32 = p.bias_kind != FA_BIAS_NONE && reinterpret_cast<uintptr_t>(p.bias) % 32 == 0 &&
                  (p.bias_stride[0] * eb) % 32 == 0 && (p.bias_stride[1] * eb) % 32 == 0 &&
                  (p.bias_stride[2] * eb) % 32 == 0;
  auto al32 = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 32 == 0 && s[0] % 16 == 0 && s[1] % 16 == 0 && s[2] % 16 == 0;
  };
  kp.ds_vec32 = al32(ds, ds_stride);
  kp.dv_vec32 = al32(p.dv, p.dv_stride);
  kp.bias = p.bias;
  kp.dv = p.dv;
  kp.lse = p.lse;
  kp.delta = p.delta;
  kp.status = status;
  kp.bias_sB = p.bias_stride[0];
  kp.bias_sH = p.bias_stride[1];
  kp.bias_sM = p.bias_stride[2];
  kp.dv_sB = p.dv_stride[0];
  kp.dv_sN = p.dv_stride[1];
  kp.dv_sH = p.dv_stride[2];
  kp.H = p.H;
  kp.M = p.M;
  kp.N = p.N;
  kp.causal = p.causal ? 1 : 0;
  kp.scale_log2 = p.sm_scale * kLog2e;
  kp.n_nblk = (p.N + 127) / 128;
  kp.n_tiles = kp.n_nblk * (slab ? slab->n_bh : p.B * p.H);
  const dim3 grid(persistent_grid(p.causal ? (kp.n_tiles + 1) / 2 : kp.n_tiles));
  r = p.dtype == FA_BF16 ? launch_bias<__nv_bfloat16>(kp, p.bias_kind, grid, stream)
                         : launch_bias<__half>(kp, p.bias_kind, grid, stream);
  return r ? r : launch_bwd_dk_from_ds(p, stream, status, slab);
}

}  // namespace fa
