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
// tile (64 KB each); Q and dO pass through a ring of three 32 KB stages, each [128 rows][128 head-dim
// columns].  Everything is kept TRANSPOSED, keys as tensor-memory lanes:
//   S^T = K Q^T, dP^T = V dO^T     (both operands in shared memory)
//   dV += P^T dO                   (P^T in tensor memory, over the columns of S^T it was formed from)
// so P needs no shared memory and the third ring stage has room.  The row threads own a key: a bias
// row, a mask row or a row of dS is then 32 neighbouring keys per warp access (64 bytes), and -LSE2 and
// -delta of the query rows come from shared memory.
// Roles (640 threads):
//   warps 0-15  row threads: lanes 32*(w&3).. (keys), 32-query column quarter w>>2
//   warps 16/17 TMA producers: each brings one of the two 16 KB boxes of every stage and half of K
//               and V (one thread's stream of boxes reaches 24 bytes per cycle, a step needs 30)
//   warp 18     MMA issuer, tensor-memory owner: per step S, dP, dV
//   warp 19     -LSE2 and -delta of a step into shared memory
// The control warps walk their loops converged and elect a lane for the issue.
// Rule kept by every barrier here: the next completion of a barrier needs progress of every thread
// that waits on it, so a parity wait can never be two phases behind.
//
// What bounds it: a step takes 6400 cycles against 3072 of products; the issuer's looks at barriers
// (200 - 235 cycles each, so they are combined) and the wait for P make up most of the rest.  (A second
// issuer for dP changed nothing: 0.245 / 0.251 ms.)  B4 H8 S2048, 16-bit bias: 0.245 ms; with the query
// rows as lanes, P in shared memory and two ring stages 0.330 ms (9800 cycles: each stage was waited for,
// and a row of bias or dS per thread is 32 sectors per warp access), with four 16 KB stages 0.379 ms
// (N = 64 products of 16-wide slices take 48 cycles, not 32, and twice the looks).
//
// Query blocks above the causal diagonal are not visited: the caller zero-fills dbias.
//
// Replaces _attn_bwd_dkdv / _attn_bwd_dkdv_inner of the reference (flash_attention.py
// 237-454) at BLOCK_HEADDIM = 256: same P, dS, dbias = dS, dK scaled by sm_scale.
#include <type_traits>

#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

struct Dkdv256Params {
  CUtensorMap map_q;   // boxes of 128 rows
  CUtensorMap map_k;
  CUtensorMap map_v;
  CUtensorMap map_do;
  CUtensorMap map_bias;  // only used to pull bias tiles into L2
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
  int causal, bias_b_mul, bias_h_mul;
  int dv_vec32;  // base and strides are multiples of 32 bytes
  float scale_log2;        // sm_scale * log2(e)
};

enum Dkdv256Site { kSiteKFull = 1, kSiteKEmpty, kSiteVFull, kSiteVEmpty, kSiteFull, kSiteEmpty, kSiteSFull,
                   kSiteStatFull, kSitePReady, kSiteDpFull, kSiteDpFree, kSiteAccDone };

constexpr int kTile256 = 128 * 256 * 2;  // K or V: four [128][64] blocks
constexpr int kStage256 = 2 * kBlk;      // [128 rows][128 columns] of Q or dO
constexpr uint32_t kStages256 = 3;
constexpr int kOffK = 0, kOffV = kOffK + kTile256, kOffRing = kOffV + kTile256;
constexpr int kSmem256 = kOffRing + kStages256 * kStage256 + 1024;  // + slack for 1024-byte alignment

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
  __shared__ uint64_t k_full, k_empty, v_full, v_empty, full[kStages256], empty[kStages256];
  __shared__ uint64_t s_full, stat_full, p_ready, dp_full, dp_free, acc_done;
  __shared__ __align__(16) float s_nlse[128], s_ndelta[128];
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
    for (uint32_t i = 0; i < kStages256; ++i) {
      mbar_init(&full[i], 2);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&stat_full, 1);
    mbar_init(&p_ready, 16);
    mbar_init(&dp_full, 1);
    mbar_init(&dp_free, 16);
    mbar_init(&acc_done, 1);
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
          const uint32_t st = use % kStages256, round = use / kStages256;
          if (round >= 1 && !wait_warp(&empty[st], (round - 1) & 1, ctx, kSiteEmpty, s.mb)) return false;
          if (elect_one()) {
            mbar_expect_tx(&full[st], kBlk);
            tma_load_4d(smem + kOffRing + st * kStage256 + half * kBlk, map, &full[st], c * 128 + half * 64, h,
                        s.mb * 128, b);
          }
          __syncwarp();
        }
        return true;
      };
      Step s;
      for (next_step(s); ok && s.valid; next_step(s)) {
        if (s.first) {
          if (nk >= 1) ok = wait_warp(&k_empty, (nk - 1) & 1, ctx, kSiteKEmpty, s.it);
          if (!ok) break;
          ++nk;
          tile_load(&p.map_k, kOffK, &k_full, s);
        }
        if (BIAS != 0 && half == 0) {
          // the bias tile of this step is pulled into L2, about a step before it is read
          constexpr int kBox = BIAS == 1 ? 64 : (BIAS == 3 ? 32 : 128);  // keys per box of map_bias
          const int b = s.bh / p.H, h = s.bh - b * p.H;
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 128; c += kBox)
              if (c == 0 || s.nb * 128 + c < p.N)
                tma_prefetch_l2_4d(&p.map_bias, s.nb * 128 + c, s.mb * 128, h * p.bias_h_mul, b * p.bias_b_mul);
          }
          __syncwarp();
        }
        ok = ring_load(&p.map_q, s);
        if (!ok) break;
        if (s.first) {
          if (nv >= 1) ok = wait_warp(&v_empty, (nv - 1) & 1, ctx, kSiteVEmpty, s.it);
          if (!ok) break;
          ++nv;
          tile_load(&p.map_v, kOffV, &v_full, s);
        }
        ok = ring_load(&p.map_do, s);
      }
    }
  } else if (warp == 18) {
    // --------------------------------------------------------------- MMA issuer
    if (live) {
      constexpr bool bf = P2::kIsBf16;
      constexpr uint32_t idesc_s = make_idesc(bf, false, false, 128, 128);
      constexpr uint32_t idesc_g = make_idesc(bf, false, true, 128, 128);
      const uint64_t k_km = make_sdesc(smem_u32(smem + kOffK), 0, 1024), v_km = make_sdesc(smem_u32(smem + kOffV), 0, 1024);
      const uint32_t ring = smem_u32(smem + kOffRing);
      constexpr uint64_t kHalfTile = static_cast<uint64_t>(2 * kBlk) >> 4;  // two blocks, in descriptor units
      bool ok = true;
      uint32_t use = 0;   // ring stages taken so far
      uint32_t tile = 0;  // K / V tiles taken so far
      uint32_t g = 0;     // steps done
      Step s;
      next_step(s);
      while (ok && s.valid) {
        const Step here = s;
        next_step(s);
        const bool last = !s.valid || s.first;  // last step of its tile
        uint32_t st[4], par[4];                 // Q and dO of this step: ring stage, parity
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          st[c] = (use + c) % kStages256;
          par[c] = ((use + c) / kStages256) & 1;
        }
        use += 4;
        // S^T: its columns hold P of the step before, whose dV this thread has issued already
        if (here.first) ok = wait_warp(&k_full, tile & 1, ctx, kSiteKFull, here.it);
        uint32_t seen0, seen1;
        mbar_poll2(&full[st[0]], par[0], &full[st[1]], par[1], seen0, seen1);
        for (int c = 0; c < 2 && ok; ++c) {
          ok = wait_warp_polled(c ? seen1 : seen0, &full[st[c]], par[c], ctx, kSiteFull, here.mb);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<8, false, false>(tmem + kColS, k_km + c * kHalfTile, make_sdesc(ring + st[c] * kStage256, 0, 1024),
                                           kBlk, kBlk, idesc_s, c > 0);
            mma_commit(&empty[st[c]]);
            if (c == 1) {
              mma_commit(&s_full);
              if (last) mma_commit(&k_empty);  // K may be replaced
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        // dP^T: its columns are free once the row threads hold dP of the step before
        if (here.first) ok = wait_warp(&v_full, tile & 1, ctx, kSiteVFull, here.it);
        uint32_t seen2 = 1;
        // (full[st[3]] is the stage of Q's first half: only asked about once S has been issued, and a
        // parity look is right then because this warp has seen that stage's completion before)
        if (g >= 1)
          mbar_poll3(&full[st[2]], par[2], &full[st[3]], par[3], &dp_free, (g - 1) & 1, seen0, seen1, seen2);
        else
          mbar_poll2(&full[st[2]], par[2], &full[st[3]], par[3], seen0, seen1);
        if (ok && g >= 1) ok = wait_warp_polled(seen2, &dp_free, (g - 1) & 1, ctx, kSiteDpFree, here.mb);
        for (int c = 0; c < 2 && ok; ++c) {
          ok = wait_warp_polled(c ? seen1 : seen0, &full[st[2 + c]], par[2 + c], ctx, kSiteFull, here.mb);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<8, false, false>(tmem + kColDp, v_km + c * kHalfTile,
                                           make_sdesc(ring + st[2 + c] * kStage256, 0, 1024), kBlk, kBlk, idesc_s, c > 0);
            if (c == 1) {
              mma_commit(&dp_full);
              if (last) mma_commit(&v_empty);
            }
          }
          __syncwarp();
        }
        if (!ok) break;
        // dV.  The first product of a tile overwrites the accumulator: P is only announced by all sixteen
        // row warps after they have read it.
        ok = wait_warp_hot(&p_ready, g & 1, ctx, kSitePReady, here.mb);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint64_t do_mn = make_sdesc(ring + st[2 + c] * kStage256, kBlk, 1024);
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)  // 16 query rows: two slices per quarter of the columns
              mma_ts(tmem + kColDv + c * 128, tmem + kColS + (ks >> 1) * 32 + (ks & 1) * 8, do_mn + mnmajor_step(ks),
                     idesc_g, !here.first || ks > 0);
            mma_commit(&empty[st[2 + c]]);
          }
          if (last) mma_commit(&acc_done);
        }
        __syncwarp();
        ++g;
        if (last) ++tile;
      }
    }
    __syncwarp();
  } else if (warp == 19) {
    // ---------------------------------------------- -LSE2 and -delta of a step's query rows
    if (live) {
      uint32_t g = 0;
      Step s;
      for (next_step(s); s.valid; next_step(s), ++g) {
        float nl[4], nd[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // rows beyond M get -inf / 0, which makes their P and dS zero
          const int m = s.mb * 128 + j * 32 + lane;
          const int64_t idx = static_cast<int64_t>(s.bh) * p.M + m;
          nl[j] = m < p.M ? -__ldcg(p.lse + idx) : -INFINITY;
          nd[j] = m < p.M ? -__ldcg(p.delta + idx) : 0.f;
        }
        if (g >= 1 && !wait_warp(&dp_free, (g - 1) & 1, ctx, kSiteDpFree, s.mb)) break;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s_nlse[j * 32 + lane] = nl[j];
          s_ndelta[j * 32 + lane] = nd[j];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&stat_full);
      }
    }
    __syncwarp();
  } else {
    // --------------------------------------------------------------- row threads
    const int r = (warp & 3) * 32 + lane;  // key inside the tile = tensor-memory lane
    const int qt = warp >> 2;              // column quarter: query rows 32*qt .. +31 of the block
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    bool ok = live;
    const uint32_t tm_sc = tmem_addr(tmem, lane_base, kColS + qt * 32);
    const uint32_t nlse_a = smem_u32(s_nlse + qt * 32), ndelta_a = smem_u32(s_ndelta + qt * 32);
    uint32_t gs = 0;     // steps done so far, over all tiles
    uint32_t tiles = 0;  // tiles with at least one step so far
    int bh, nb, i_start;
#pragma unroll 1
    for (int it = 0; ok && tile_at(it, bh, nb, i_start); ++it) {
      const int n = nb * 128 + r;
      const int b = bh / p.H, h = bh - b * p.H;
      const bool key_ok = n < p.N;
      // Keys beyond N compute on zero rows of K and V and what they read as bias is key N-1's; nothing of
      // theirs is stored, and no other key's result depends on them.
      const int64_t bias_off = b * p.bias_sB + h * p.bias_sH + min(n, p.N - 1);
      const int64_t ds_off = (p.ds_flat ? (bh - p.bh0) * p.ds_sH : b * p.ds_sB + h * p.ds_sH) + n;
      const int64_t dbf_off = b * p.dbf_sB + h * p.dbf_sH + n;
#pragma unroll 1
      for (int mb = i_start; mb < n_mblk && ok; ++mb, ++gs) {
        const int m0 = mb * 128 + qt * 32;  // this thread's first query row
        const int rows = p.M - m0;          // of its 32 query rows the first `rows` exist
        // The bias of this step travels while S is computed.  (Whole blocks without a test per row: with
        // one the loads went out one after the other, 8200 cycles a step.)
        uint32_t w[BIAS != 0 ? 32 : 1];
        if constexpr (BIAS != 0) {
          using E = std::conditional_t<BIAS == 1, uint16_t, std::conditional_t<BIAS == 2, uint8_t, uint32_t>>;
          const E* src = static_cast<const E*>(p.bias) + bias_off;
          if (rows >= 32) {
            src += static_cast<int64_t>(m0) * p.bias_sM;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              w[i] = __ldcg(src);
              src += p.bias_sM;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              w[i] = __ldcg(src + static_cast<int64_t>(min(m0 + i, p.M - 1)) * p.bias_sM);
              if (i >= rows) w[i] = 0;
            }
          }
        }

        // ---- P^T
        uint32_t ps, pstat;
        mbar_poll2(&s_full, gs & 1, &stat_full, gs & 1, ps, pstat);
        ok = wait_warp_polled(pstat, &stat_full, gs & 1, ctx, kSiteStatFull, mb);
        if (ok) ok = wait_warp_polled(ps, &s_full, gs & 1, ctx, kSiteSFull, mb);
        if (!ok) break;
        tc_fence_after();
        float pr[32];
        tmem_ld32(tm_sc, reinterpret_cast<uint32_t*>(pr));
        tmem_ld_wait();
        // P = exp2(S * scale * log2e + bias * log2e - LSE2)
        const f32x2 sc2 = f2(p.scale_log2, p.scale_log2);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 v = lds128(nlse_a + c * 16);
          const f32x2 nl[2] = {f2(__uint_as_float(v.x), __uint_as_float(v.y)), f2(__uint_as_float(v.z), __uint_as_float(v.w))};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = c * 4 + e * 2;
            f32x2 a = ffma2(f2(pr[i], pr[i + 1]), sc2, nl[e]);
            if constexpr (BIAS == 1) {
              const float2 f = P2::unpack(w[i] | (w[i + 1] << 16));
              a = ffma2(f2(f.x, f.y), f2(kLog2e, kLog2e), a);
            } else if constexpr (BIAS == 3) {
              a = ffma2(f2(__uint_as_float(w[i]), __uint_as_float(w[i + 1])), f2(kLog2e, kLog2e), a);
            }
            pr[i] = ex2(f2_lo(a));
            pr[i + 1] = ex2(f2_hi(a));
            if constexpr (BIAS == 2) {
              pr[i] = w[i] != 0 ? pr[i] : 0.f;
              pr[i + 1] = w[i + 1] != 0 ? pr[i + 1] : 0.f;
            }
          }
        }
        if (p.causal && nb * 128 + 127 > m0) {
          const int hidden = n - m0;  // the first query rows do not see this key
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < hidden) pr[i] = 0.f;
        }
        {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = P2::pack(pr[2 * i], pr[2 * i + 1]);
          tmem_st16(tm_sc, pk);  // over this thread's own scores
          tmem_st_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready);

        // ---- dS = P * (dP - delta)
        ok = wait_warp(&dp_full, gs & 1, ctx, kSiteDpFull, mb);
        if (!ok) break;
        tc_fence_after();
        uint32_t all = 0xffffffffu;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t dp[16];
          tmem_ld16(tm_sc + (kColDp - kColS) + hf * 16, dp);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint4 v = lds128(ndelta_a + hf * 64 + c * 16);
            const f32x2 nd[2] = {f2(__uint_as_float(v.x), __uint_as_float(v.y)), f2(__uint_as_float(v.z), __uint_as_float(v.w))};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int k = c * 4 + e * 2, i = hf * 16 + k;
              const f32x2 d = fmul2(f2(pr[i], pr[i + 1]),
                                    fadd2(f2(__uint_as_float(dp[k]), __uint_as_float(dp[k + 1])), nd[e]));
              pr[i] = f2_lo(d);
              pr[i + 1] = f2_hi(d);
              all &= __float_as_uint(pr[i]) & __float_as_uint(pr[i + 1]);
            }
          }
        }
        // dP and the row statistics go back only once every lane has used them (the vote needs them all)
        if (__all_sync(0xffffffffu, all == 0xffffffffu)) tc_fence_after();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&dp_free);
        if (key_ok) {
          uint16_t* drow = static_cast<uint16_t*>(p.ds16) + ds_off + static_cast<int64_t>(m0) * p.ds_sM;
          if (rows >= 32) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const uint32_t d2 = P2::pack(pr[i], pr[i + 1]);
              drow[0] = static_cast<uint16_t>(d2);
              drow[p.ds_sM] = static_cast<uint16_t>(d2 >> 16);
              drow += 2 * p.ds_sM;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const uint32_t d2 = P2::pack(pr[i], pr[i + 1]);
              if (i < rows) drow[i * p.ds_sM] = static_cast<uint16_t>(d2);
              if (i + 1 < rows) drow[(i + 1) * p.ds_sM] = static_cast<uint16_t>(d2 >> 16);
            }
          }
          if (BIAS == 3 && p.dbias_f32 != nullptr) {
            // the fp32 bias gradient goes out unrounded
            float* frow = p.dbias_f32 + dbf_off + static_cast<int64_t>(m0) * p.dbf_sM;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (i < rows) frow[i * p.dbf_sM] = pr[i];
          }
        }
      }
      if (!ok) break;

      // ---- epilogue: dV (rows = keys) -> global, 64 head-dim columns per thread
      const bool any = i_start < n_mblk;
      if (any) {
        ok = wait_warp(&acc_done, tiles & 1, ctx, kSiteAccDone, it);
        if (!ok) break;
        ++tiles;
      }
      tc_fence_after();
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
        if (key_ok) {
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
  auto al32 = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 32 == 0 && s[0] % 16 == 0 && s[1] % 16 == 0 && s[2] % 16 == 0;
  };
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
