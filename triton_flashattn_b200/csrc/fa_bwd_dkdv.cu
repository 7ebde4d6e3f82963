// dK / dV (and dbias) kernel for sm_100a.
//
// Persistent kernel, one CTA per SM.  A tile is 128 keys of one (batch, head); a CTA
// walks its tiles one after the other and, inside a tile, the query blocks of 128 rows
// (only those at or below the diagonal when causal).  Ring stages, tensor-memory buffers
// and barrier phases run on from tile to tile, so the next tile's K / V / Q / dO loads,
// its first S and dP products and its first bias rows overlap the current tile's
// epilogue.  Roles (384 threads):
//   warps 0-7  "row" threads: warp w works on tensor-memory lanes 32*(w&3)..+31
//              (query rows of the block) and on the 64-key half (w>>2)
//   warp 8     TMA producer: K, V per tile; Q ring (2), dO ring; bias tiles: loaded, or asked
//              into L2 one step ahead, or (16 bit at head dim 128) both
//   warp 9     MMA issuer for S and dP, tensor-memory owner
//   warp 10    MMA issuer for dV and dK
//   warp 11    bulk tensor stores of dS (into dbias or scratch)
// The four control warps walk their loops with all lanes converged and elect a lane only
// for the TMA / MMA / commit instructions, whose operands are then warp-uniform values.
// A wait takes 200 - 235 cycles here even on a completed barrier, so two issuers keep
// the tensor pipe fed while the other one waits, each looks at the barriers of a product together, and the row threads
// ask for the barriers they will need before the fence that ends the stretch before.  Whole backward, us, before these
// looks and a warp of their own for the stores (which held the dV / dK issuer up until dS was read) / after: no bias
// B2 H16 S4096 D64 683 / 636, B4 H16 S2048 D128 411 / 400; 16 bit B8 H16 S2048 D64 758 / 728.
// Per query block t:
//   S  = Q_t K^T            (tensor memory, 128 columns)
//   dP = dO_t V^T           (tensor memory, 128 columns)
//   row threads: P = exp2(S*scale*log2e + bias*log2e - LSE2) -> 16-bit tile sP
//                dS = P * (dP - delta)                        -> 16-bit tile sDS
//   dV += P^T dO_t          (sP and dO_t consumed MN-major)
//   dK += dS^T Q_t          (sDS and Q_t consumed MN-major)
//   dbias[b,h,m-block,n-block] <- sDS  (one bulk tensor store of the same tile)
// Bias.  16 bit, and a mask at head dim 64: by TMA, at head dim 64 into two tiles of its own, at 128, where no shared memory
// is left, exactly where the row threads then write P: each thread reads the eight 16-byte chunks it is about to
// overwrite.  (Read by the row threads into registers a step ahead it takes no part in the chain of a step, but a load of 32
// rows costs 24 - 60 cycles to issue: 5 - 12 % slower.)  A mask at head dim 128 and an fp32 bias are read by the row threads
// straight from global memory, the mask 64 contiguous bytes per thread, one query block ahead.
// Causally skipped tiles of dbias are written as zeros by this kernel, so dbias
// needs no prior fill.
// Rule kept by every barrier here: the next completion of a barrier needs progress of
// every thread that waits on it, so a parity wait can never be two phases behind.
//
// With at most 128 keys one tile holds a whole row of dS, and the ONE_TILE variant (head dims up to 64, up to 256 queries)
// is the whole backward in one launch: dQ = dS K over the tile of dS that dK reads, into 64 free columns of tensor memory,
// and delta from the rows of o and dO, which the threads of that query row add up as fa_bwd_pre.cu does (the same bits).
// It saves two launches, and with an fp32 bias the way of dS through memory (it is only stored for a caller that gives
// a ds16), but a tile's chain is longer (see
// one_tile_takes).
//
// Replaces _attn_bwd_dkdv / _attn_bwd_dkdv_inner of the reference
// (flash_attention.py 237-454): same P, dS, dbias = dS, dK scaled by sm_scale.
#include "fa_common.cuh"
#include "fa_host.cuh"

namespace fa {
namespace {

struct DkdvParams {
  CUtensorMap map_q;
  CUtensorMap map_k;
  CUtensorMap map_v;
  CUtensorMap map_do;
  CUtensorMap map_dbias;
  CUtensorMap map_bias;  // tiles of a 16-bit bias and, at head dim 64, of a mask; the others are only asked into L2 through it
  const void* bias;
  void* dk;
  void* dv;
  const float* lse;
  const float* delta;
  int* status;
  int64_t bias_sB, bias_sH, bias_sM;
  int64_t dk_sB, dk_sN, dk_sH, dv_sB, dv_sN, dv_sH;
  int H, M, N, D;
  int n_nblk, n_tiles;  // key blocks per (batch, head); tiles of this launch
  int bh0;              // first (batch, head) of this launch
  int ds_flat;          // dS goes to slabs numbered from bh0 instead of a (B, H, M, N) tensor
  int causal, bias_vec32, bias_b_mul, bias_h_mul;
  int dkv_vec32;  // dk / dv bases and strides are multiples of 32 bytes
  int store_ds;    // the 16-bit dS tiles go out through map_dbias (as dbias, or as scratch for dQ)
  int zero_tiles;  // ... and zero tiles go to the causally skipped part (16-bit dbias only)
  float* dbias_f32;  // fp32 bias gradient, written from registers (fp32 bias only), or null
  int64_t dbf_sB, dbf_sH, dbf_sM;
  float scale_log2;  // sm_scale * log2(e)
  float sm_scale;
  int n_bh;  // problems of this launch
  // one tile of keys: what dQ and delta need
  const void* o;
  const void* d_o;
  void* dq;
  float* delta_out;
  int64_t o_sB, o_sM, o_sH, do_sB, do_sM, do_sH, dq_sB, dq_sM, dq_sH;
};

enum DkdvSite { kSiteKV = 1, kSiteQFull, kSiteQEmpty, kSiteDoFull, kSiteDoEmpty, kSiteSFull,
                kSiteDpFull, kSitePReady, kSiteDsReady, kSiteDvDone, kSiteDkDone, kSiteStDone,
                kSiteZeroReady, kSiteEpilogue, kSiteSFree, kSiteDpFree, kSiteKVEmpty, kSiteBiasFull, kSiteBiasEmpty };

// Eight row warps, a thread with half a row of a step: what a step costs a warp besides its values (looks at nine
// barriers, votes, fences, loop) is paid half as often as with sixteen warps and quarters of a row, and 168 registers
// hold the rest, but for ONE_TILE: its eight chunks each of o and dO, asked for ahead of a step, spill (bytes stored / loaded:
// no bias 66 / 96, 16 bit 150 / 304, mask 102 / 168, fp32 338 / 480; the other variants 4 / 16 at most).  Whole backward, us, quarters / halves: no bias B4 H16 S2048 D128 403 / 400, 16 bit B8 H16 S2048 D128 902 / 894,
// D64 742 / 728, mask, causal, B4 H32 S4096 D128 1805 / 1754, fp32 B4 H16 S2048 D128 882 / 867.
constexpr int kCW = 64;           // columns of a step that a row thread works on
constexpr int kNG = kCW / 32;     // ... in groups of 32
constexpr int kRW = 512 / kCW;    // row warps
constexpr int kThreads = 32 * (kRW + 4);
template <int DP, int BIAS>
struct DkdvSmem {
  static constexpr int kTile = 128 * DP * 2;
  static constexpr int kDoStages = DP == 128 ? 1 : 2;
  static constexpr int kK = 0;
  static constexpr int kV = kK + kTile;
  static constexpr int kQ = kV + kTile;
  static constexpr int kDo = kQ + 2 * kTile;
  static constexpr int kP = kDo + kDoStages * kTile;
  static constexpr int kDs = kP + 2 * kBlk;
  // At head dim 64 there is room for two tiles of a 16-bit bias or a mask of their own, which then land a step ahead and
  // not between two steps (16 bit) or load by load through the row threads (mask).  Whole backward, us, before / after: 16
  // bit, trained, B8 H16 S2048 722 / 687, causal 508 / 488, B32 H16 S512 239 / 226; mask B8 H12 S1000 227 / 203, B2 H16 S4096
  // 654 / 638.
  static constexpr bool kOwnBias = DP == 64 && (BIAS == 1 || BIAS == 2);
  static constexpr int kBiasTile = BIAS == 1 ? 2 * kBlk : kBlk;
  static constexpr int kBias = kDs + 2 * kBlk;
  static constexpr int kTotal = kBias + (kOwnBias ? 2 * kBiasTile : 0);
  static constexpr int kDynamic = kTotal + 1024;
};

template <int DP, typename T, int BIAS, bool LONGEST_FIRST, bool ONE_TILE = false>
__global__ void __launch_bounds__(kThreads, 1) dkdv_kernel(const __grid_constant__ DkdvParams p) {
  using L = DkdvSmem<DP, BIAS>;
  using P2 = Pack2<T>;
  constexpr int KB = DP / 64;
  constexpr int KS_D = DP / 16;  // K slices of the two "score" products
  constexpr int kDoStages = L::kDoStages;
  constexpr uint32_t kColS = 0, kColDp = 128, kColDv = 256, kColDk = 384;
  constexpr uint32_t kColDq = 320;  // one tile of keys, head dims up to 64
  static_assert(!ONE_TILE || (DP == 64 && !LONGEST_FIRST), "dQ has no columns");
  constexpr uint32_t kTmemCols = 512;
  // BIAS: 0 none; 1 16-bit bias; 2 byte mask; 3 fp32 bias (its row - 64 registers - is asked for at the start of its own step)
  constexpr int BK = BIAS;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  __shared__ uint64_t kv_full, kv_empty, q_full[2], q_empty[2], do_full[2], do_empty[2];
  __shared__ uint64_t s_full, dp_full, p_ready, ds_ready, dv_done, dk_done, st_done, zero_ready;
  __shared__ uint64_t s_free, dp_free, bias_full[2], bias_empty[2];  // bias: one tile (in sP), or two of its own
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int tid = threadIdx.x;
  // the warp index as a value the compiler knows to be the same in all lanes: the role
  // branches below are then warp-uniform and the issuer warps run converged
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int n_mblk = (p.M + 127) >> 7;

  // Schedule: tiles are numbered (batch*head)-major; CTA c takes units c, c+G, c+2G, ... so
  // that CTAs running at the same time work on neighbouring tiles and share Q / dO in L2.  A
  // unit is one tile, or - causal - two consecutive entries of the per-(batch, head) order
  // [first, last, first+1, last-1, ...]: a heavy and a light key block.
  // With LONGEST_FIRST (causal, few tiles a CTA) the tiles are numbered by length instead, and the CTAs take them in rows,
  // every second row from the other end: what a CTA has too much of in one row it has too little of in the next.  It is a
  // variant of its own because every role walks the schedule: chosen at run time it cost every short tile of the others
  // (trained bias shared by the batch, 72 x 72, B539 H3 D16 44.4 -> 49.0 us, 100 x 100, B600 H4 D64 69.0 -> 74.3).
  const int sched_sh = p.causal && !ONE_TILE ? 1 : 0;
  auto tile_at = [&](int it, int& bh, int& nb, int& i_start, int& T_steps) -> bool {
    if constexpr (LONGEST_FIRST) {
      const int G = static_cast<int>(gridDim.x), c = static_cast<int>(blockIdx.x);
      const int k = it * G + ((it & 1) ? G - 1 - c : c);
      if (k >= p.n_tiles) return false;
      nb = k / p.n_bh;
      bh = p.bh0 + k - nb * p.n_bh;
      i_start = min(nb, n_mblk);
      T_steps = n_mblk - i_start;
      return true;
    }
    const int u = static_cast<int>(blockIdx.x) + (it >> sched_sh) * static_cast<int>(gridDim.x);
    const int k = (u << sched_sh) + (it & sched_sh);
    if (k >= p.n_tiles) return false;
    bh = k / p.n_nblk;
    const int pos = k - bh * p.n_nblk;
    bh += p.bh0;
    nb = sched_sh ? ((pos & 1) ? p.n_nblk - 1 - (pos >> 1) : (pos >> 1)) : pos;
    i_start = p.causal ? min(nb, n_mblk) : 0;
    T_steps = n_mblk - i_start;
    return true;
  };

  WaitCtx ctx{&abort_flag, p.status, 2};

  if (tid == 0) {
    abort_flag = 0;
    mbar_init(&kv_full, 1);
    mbar_init(&kv_empty, ONE_TILE ? 2 : 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 2);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 2);
    }
    mbar_init(&s_full, 1);
    mbar_init(&dp_full, 1);
    mbar_init(&p_ready, kRW);
    mbar_init(&ds_ready, kRW);
    mbar_init(&dv_done, 1);
    mbar_init(&dk_done, 1);
    mbar_init(&st_done, 1);
    mbar_init(&zero_ready, kRW);
    mbar_init(&s_free, kRW);
    mbar_init(&dp_free, kRW);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bias_full[i], 1);
      mbar_init(&bias_empty[i], kRW);
    }
    mbar_fence_init();
  }
  if (warp == kRW + 1) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  grid_dep_launch_next();
  grid_dep_wait();  // the previous kernel's results (and its status word) are visible from here
  const bool live = *reinterpret_cast<volatile int*>(p.status) == 0;

  if (warp == kRW) {
    // ------------------------------------------------------------------ producer
    // (whole warp converged, one elected lane issues)
    if (live) {
      if (lane == 0) {
        tma_prefetch_desc(&p.map_q);
        tma_prefetch_desc(&p.map_k);
        tma_prefetch_desc(&p.map_v);
        tma_prefetch_desc(&p.map_do);
      }
      bool ok = true;
      constexpr int kBiasAhead = 1;  // bias tiles are pulled into L2 this many steps early
      uint32_t g = 0;                // steps issued so far, over all tiles
      uint32_t kvi = 0;              // tiles with at least one step so far
      int pf_done = 0;               // bias tiles of the coming tile already requested
      int bh, nb, i_start, T_steps;
      for (int it = 0; ok && tile_at(it, bh, nb, i_start, T_steps); ++it) {
        if (T_steps <= 0) continue;
        const int b = bh / p.H, h = bh - b * p.H, n0 = nb * 128;
        // K and V are single tiles: free once the previous tile's last S and dP are through
        if (kvi >= 1) ok = wait_warp(&kv_empty, (kvi - 1) & 1, ctx, kSiteKVEmpty, it);
        if (!ok) break;
        ++kvi;
        if (elect_one()) {
          mbar_expect_tx(&kv_full, 2 * L::kTile);
          for (int kb = 0; kb < KB; ++kb) {
            tma_load_4d(smem + L::kK + kb * kBlk, &p.map_k, &kv_full, kb * 64, h, n0, b);
            tma_load_4d(smem + L::kV + kb * kBlk, &p.map_v, &kv_full, kb * 64, h, n0, b);
          }
        }
        __syncwarp();
        // Bias tiles are pulled into L2 kBiasAhead steps before the row threads read them,
        // as one stream over tile boundaries: the last steps of a tile request the first
        // tiles of the next one (pf_done of them are out when that tile starts).
        auto bias_l2 = [&](int b_, int h_, int n0_, int mblk) {
          const int mp = mblk * 128;
          constexpr int kBox = BK == 1 ? 64 : (BK == 3 ? 32 : 128);  // keys per box of map_bias
          if (elect_one()) {
#pragma unroll
            for (int c = 0; c < 128; c += kBox)
              if (c == 0 || n0_ + c < p.N)
                tma_prefetch_l2_4d(&p.map_bias, n0_ + c, mp, h_ * p.bias_h_mul, b_ * p.bias_b_mul);
          }
          __syncwarp();
        };
        constexpr bool kAskL2 = BIAS != 0 && !L::kOwnBias;
        if (kAskL2) {
          for (int t = pf_done; t < kBiasAhead && t < T_steps; ++t) bias_l2(b, h, n0, i_start + t);
          pf_done = 0;
        }
        int bh2 = 0, nb2 = 0, is2 = 0, T2 = 0;
        if (kAskL2 && !tile_at(it + 1, bh2, nb2, is2, T2)) T2 = 0;
        for (int t = 0; t < T_steps && ok; ++t) {
          const uint32_t gs = g + t;
          const int m0 = (i_start + t) * 128;
          const int qs = gs & 1;
          if (kAskL2) {
            if (t + kBiasAhead < T_steps) {
              bias_l2(b, h, n0, i_start + t + kBiasAhead);
            } else if (t + kBiasAhead - T_steps < T2) {
              const int b2 = bh2 / p.H;
              bias_l2(b2, bh2 - b2 * p.H, nb2 * 128, is2 + t + kBiasAhead - T_steps);
              ++pf_done;
            }
          }
          if constexpr (L::kOwnBias) {
            // two steps ahead of the row threads at the most
            if (gs >= 2) ok = wait_warp(&bias_empty[qs], ((gs >> 1) - 1) & 1, ctx, kSiteBiasEmpty, t);
            if (!ok) break;
            const bool two = BIAS == 1 && n0 + 64 < p.N;
            if (elect_one()) {
              uint8_t* const dst = smem + L::kBias + qs * L::kBiasTile;
              mbar_expect_tx(&bias_full[qs], two ? 2 * kBlk : kBlk);
              tma_load_4d(dst, &p.map_bias, &bias_full[qs], n0, m0, h * p.bias_h_mul, b * p.bias_b_mul);
              if (two) tma_load_4d(dst + kBlk, &p.map_bias, &bias_full[qs], n0 + 64, m0, h * p.bias_h_mul, b * p.bias_b_mul);
            }
            __syncwarp();
          }
          if (gs >= 2) ok = wait_warp(&q_empty[qs], ((gs >> 1) - 1) & 1, ctx, kSiteQEmpty, t);
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(&q_full[qs], L::kTile);
            for (int kb = 0; kb < KB; ++kb)
              tma_load_4d(smem + L::kQ + qs * L::kTile + kb * kBlk, &p.map_q, &q_full[qs], kb * 64, h,
                          m0, b);
          }
          __syncwarp();
          // The [128 rows][128 keys] 16-bit bias tile of a step lands exactly where the row threads
          // will then write P (same two swizzled blocks, every thread reads the 16-byte
          // chunks it is about to overwrite): no extra shared memory.  sP is free for it once the
          // dV product of the previous step has read P, which at head dim 128 also frees dO.
          auto load_bias = [&]() {
            if (gs >= 1) ok = wait_warp_hot(&dv_done, (gs - 1) & 1, ctx, kSiteDvDone, t);
            if (!ok) return;
            const bool two = n0 + 64 < p.N;
            if (elect_one()) {
              mbar_expect_tx(&bias_full[0], two ? 2 * kBlk : kBlk);
              tma_load_4d(smem + L::kP, &p.map_bias, &bias_full[0], n0, m0, h * p.bias_h_mul, b * p.bias_b_mul);
              if (two)
                tma_load_4d(smem + L::kP + kBlk, &p.map_bias, &bias_full[0], n0 + 64, m0, h * p.bias_h_mul,
                            b * p.bias_b_mul);
            }
            __syncwarp();
          };
          if (BIAS == 1 && !L::kOwnBias) load_bias();
          if (!ok) break;
          const int ds = gs % kDoStages;
          const uint32_t du = gs / kDoStages;
          if (du >= 1) ok = wait_warp(&do_empty[ds], (du - 1) & 1, ctx, kSiteDoEmpty, t);
          if (!ok) break;
          if (elect_one()) {
            mbar_expect_tx(&do_full[ds], L::kTile);
            for (int kb = 0; kb < KB; ++kb)
              tma_load_4d(smem + L::kDo + ds * L::kTile + kb * kBlk, &p.map_do, &do_full[ds], kb * 64,
                          h, m0, b);
          }
          __syncwarp();
        }
        g += T_steps;
      }
    }
  } else if (warp == kRW + 1) {
    // ------------------------------------------------------- MMA issuer: S and dP
    // The whole warp walks the loop (waits included) and one elected lane issues: the
    // descriptors are then warp-uniform values, which the tensor-core instructions take
    // without a per-operand transfer from a lane's registers.
    if (live) {
      constexpr bool bf = P2::kIsBf16;
      constexpr uint32_t idesc_s = make_idesc(bf, false, false, 128, 128);
      const uint32_t k_addr = smem_u32(smem + L::kK), v_addr = smem_u32(smem + L::kV);
      const uint32_t q_addr = smem_u32(smem + L::kQ), do_addr = smem_u32(smem + L::kDo);
      const uint64_t k_km = make_sdesc(k_addr, 0, 1024), v_km = make_sdesc(v_addr, 0, 1024);
      const uint64_t q_km_0 = make_sdesc(q_addr, 0, 1024), q_km_1 = make_sdesc(q_addr + L::kTile, 0, 1024);
      const uint64_t do_km_0 = make_sdesc(do_addr, 0, 1024),
                     do_km_1 = make_sdesc(do_addr + (kDoStages - 1) * L::kTile, 0, 1024);
      bool ok = true;
      uint32_t g = 0, kvi = 0;
      int bh, nb, i_start, T_steps;
      for (int it = 0; ok && tile_at(it, bh, nb, i_start, T_steps); ++it) {
        if (T_steps <= 0) continue;
        ok = wait_warp(&kv_full, kvi & 1, ctx, kSiteKV, it);
        ++kvi;
        for (int t = 0; t < T_steps && ok; ++t) {
          const uint32_t gs = g + t;
          const int qs = gs & 1, ds = gs % kDoStages;
          const uint32_t q_par = (gs >> 1) & 1, do_par = (gs / kDoStages) & 1;
          // S_gs: its columns are free once the row threads hold S_{gs-1} in registers
          ok = gs >= 1 ? wait_all2<false>(&s_free, (gs - 1) & 1, &q_full[qs], q_par, ctx, kSiteSFree, t)
                       : wait_all1<false>(&q_full[qs], q_par, ctx, kSiteQFull, t);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<KS_D, false, false>(tmem + kColS, qs ? q_km_1 : q_km_0, k_km, kBlk, kBlk,
                                              idesc_s, false);
            mma_commit(&s_full);
            mma_commit(&q_empty[qs]);
          }
          // dP_gs: same for the dP columns; dO_gs replaces dO_{gs-1} after dV_{gs-1} when
          // single-staged
          ok = gs >= 1 ? wait_all2<false>(&dp_free, (gs - 1) & 1, &do_full[ds], do_par, ctx, kSiteDpFree, t)
                       : wait_all1<false>(&do_full[ds], do_par, ctx, kSiteDoFull, t);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<KS_D, false, false>(tmem + kColDp, ds ? do_km_1 : do_km_0, v_km, kBlk, kBlk,
                                              idesc_s, false);
            mma_commit(&dp_full);
            mma_commit(&do_empty[ds]);
            if (t == T_steps - 1) mma_commit(&kv_empty);  // K and V may be replaced
          }
        }
        g += T_steps;
      }
    }
    __syncwarp();
  } else if (warp == kRW + 2) {
    // ------------------------------------------------------ MMA issuer: dV and dK
    // (whole warp converged, one elected lane issues: see the S / dP issuer)
    if (live) {
      constexpr bool bf = P2::kIsBf16;
      constexpr uint32_t idesc_g = make_idesc(bf, true, true, 128, DP);
      const uint32_t q_addr = smem_u32(smem + L::kQ), do_addr = smem_u32(smem + L::kDo);
      const uint32_t p_addr = smem_u32(smem + L::kP), ds_addr = smem_u32(smem + L::kDs);
      const uint64_t q_mn_0 = make_sdesc(q_addr, kBlk, 1024), q_mn_1 = make_sdesc(q_addr + L::kTile, kBlk, 1024);
      const uint64_t do_mn_0 = make_sdesc(do_addr, kBlk, 1024),
                     do_mn_1 = make_sdesc(do_addr + (kDoStages - 1) * L::kTile, kBlk, 1024);
      const uint64_t p_mn = make_sdesc(p_addr, kBlk, 1024), ds_mn = make_sdesc(ds_addr, kBlk, 1024);
      bool ok = true;
      uint32_t g = 0;
      int bh, nb, i_start, T_steps;
      for (int it = 0; ok && tile_at(it, bh, nb, i_start, T_steps); ++it) {
        for (int t = 0; t < T_steps && ok; ++t) {
          const uint32_t gs = g + t;
          const int qs = gs & 1;
          const int ds = gs % kDoStages;
          // dV += P^T dO  (dO must have landed: P only depends on S).  The first product of a
          // tile overwrites dV / dK: P and dS of a new tile are only announced by all eight
          // row warps after they have read the previous tile's accumulators.
          ok = wait_all2<false>(&p_ready, gs & 1, &do_full[ds], (gs / kDoStages) & 1, ctx, kSitePReady, t);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<8, true, true>(tmem + kColDv, p_mn, ds ? do_mn_1 : do_mn_0, kBlk, kBlk, idesc_g,
                                         t > 0);
            mma_commit(&dv_done);
            mma_commit(&do_empty[ds]);
          }
          // dK += dS^T Q
          ok = wait_all2<false>(&ds_ready, gs & 1, &q_full[qs], (gs >> 1) & 1, ctx, kSiteDsReady, t);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            issue_gemm_ss<8, true, true>(tmem + kColDk, ds_mn, qs ? q_mn_1 : q_mn_0, kBlk, kBlk, idesc_g,
                                         t > 0);
            if constexpr (ONE_TILE) {
              // its columns are free: dS is only announced by row warps that have read the dQ of the step before
              issue_gemm_ss<8, false, true>(tmem + kColDq, make_sdesc(ds_addr, 0, 1024), make_sdesc(smem_u32(smem + L::kK), kBlk, 1024),
                                            kBlk, kBlk, make_idesc(bf, false, true, 128, DP), false);
              if (t == T_steps - 1) mma_commit(&kv_empty);
            }
            mma_commit(&q_empty[qs]);
            mma_commit(&dk_done);
          }
        }
        g += T_steps;
      }
    }
    __syncwarp();
  } else if (warp == kRW + 3) {
    // ----------------------------------------------------------- stores of dS
    // (whole warp converged, one elected lane issues)
    // st_done completes once per step when the store of dS has finished reading sDS and - where there are zero tiles -
    // once per tile before that, when those above the diagonal are out.  (Without the zero tiles there is no per-tile
    // completion: two completions in a row that no row thread has to wait for in between would let a parity wait fall
    // two phases behind.)
    if (live && p.store_ds) {
      if (lane == 0) tma_prefetch_desc(&p.map_dbias);
      bool ok = true;
      uint32_t g = 0;
      int bh, nb, i_start, T_steps;
      for (int it = 0; ok && tile_at(it, bh, nb, i_start, T_steps); ++it) {
        const int b = bh / p.H, h = bh - b * p.H, n0 = nb * 128;
        const int ds_h = p.ds_flat ? bh - p.bh0 : h, ds_b = p.ds_flat ? 0 : b;
        const bool two = n0 + 64 < p.N;
        if (p.zero_tiles) {
          ok = wait_warp(&zero_ready, it & 1, ctx, kSiteZeroReady, it);
          if (!ok) break;
          if (elect_one()) {
            for (int i = 0; i < i_start; ++i) {
              tma_store_4d(&p.map_dbias, smem + L::kDs, n0, i * 128, h, b);
              if (two) tma_store_4d(&p.map_dbias, smem + L::kDs + kBlk, n0 + 64, i * 128, h, b);
            }
            tma_store_commit();
            tma_store_wait_read<0>();
            mbar_arrive(&st_done);
          }
          __syncwarp();
        }
        for (int t = 0; t < T_steps && ok; ++t) {
          // (Right when dS is there the store competes with dK for shared memory: D128, mask, causal B4 H32 S4096 1764 ->
          // 1893 us, 16-bit bias B8 H16 S2048 898 -> 910.)
          ok = wait_warp(&dk_done, (g + t) & 1, ctx, kSiteDkDone, t);
          if (!ok) break;
          const int m0 = (i_start + t) * 128;
          if (elect_one()) {
            tma_store_4d(&p.map_dbias, smem + L::kDs, n0, m0, ds_h, ds_b);
            if (two) tma_store_4d(&p.map_dbias, smem + L::kDs + kBlk, n0 + 64, m0, ds_h, ds_b);
            tma_store_commit();
            tma_store_wait_read<0>();
            mbar_arrive(&st_done);
          }
          __syncwarp();
        }
        g += T_steps;
      }
      if (elect_one()) tma_store_wait_all<0>();
    }
    __syncwarp();
  } else {
    // --------------------------------------------------------------- row threads
    const int r = (warp & 3) * 32 + lane;  // query row inside the block = tensor-memory lane
    const int qt = warp >> 2;              // column group: keys n0 + kCW*qt .. + kCW-1
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    bool ok = live;
    // this thread's eight 16-byte chunks inside the [128][128] 16-bit tiles: chunk c of the
    // row lands at sp_row + ((chunk0 + c) ^ (r & 7)) * 16; the dS tile sits kDs - kP further
    const uint32_t sp_row = smem_u32(smem + L::kP + (qt * kCW / 64) * kBlk) + static_cast<uint32_t>(r) * 128u;
    const uint32_t chunk0 = (qt * kCW % 64) / 8;
    // tensor-memory address of this thread's 64 columns of S (dP: + kColDp)
    const uint32_t tm_sc = tmem_addr(tmem, lane_base, kColS + qt * kCW);

    constexpr int BR = BIAS == 1 || L::kOwnBias ? 0 : BK;  // bias read by the row threads: fp32, and a mask without tiles of its own
    constexpr bool kBiasTma = BIAS == 1 || L::kOwnBias;
    constexpr bool kBiasInP = kBiasTma && !L::kOwnBias;
    BiasRegs<BR> bnext[kNG];
    // LSE2 and delta of the coming step's row, as loaded: they are only looked at (negated,
    // replaced for rows beyond M) when that step starts, so the loads travel during this one
    float lse_next = 0.f, delta_next = 0.f;
    bool row_ok_next = false;
    uint4 o_next[ONE_TILE ? 8 : 1], do_next[ONE_TILE ? 8 : 1];  // delta is formed from them instead
    // fetches bias / -LSE2 / delta of query block `mblk` for the tile (bh_, key column c0)
    auto prefetch = [&](int bh_, int c0, int mblk) {
      const int b_ = bh_ / p.H, h_ = bh_ - b_ * p.H;
      const int64_t bias_bh = b_ * p.bias_sB + h_ * p.bias_sH;
      const int m = mblk * 128 + r;
      const bool row_ok = m < p.M;
      if constexpr (BR == 2) {
#pragma unroll
        for (int g = 0; g < kNG; ++g)
          load_bias_row<BK>(bnext[g], p.bias, bias_bh + (int64_t)m * p.bias_sM, row_ok, c0 + g * 32, p.N,
                            p.bias_vec32 != 0);
      }
      const int64_t idx = (int64_t)bh_ * p.M + min(m, p.M - 1);
      lse_next = __ldcg(p.lse + idx);
      row_ok_next = row_ok;
      if constexpr (!ONE_TILE) {
        delta_next = __ldcg(p.delta + idx);
      } else {
        const uint4* orow = reinterpret_cast<const uint4*>(static_cast<const T*>(p.o) + b_ * p.o_sB + (int64_t)min(m, p.M - 1) * p.o_sM +
                                                           h_ * p.o_sH);
        const uint4* grow = reinterpret_cast<const uint4*>(static_cast<const T*>(p.d_o) + b_ * p.do_sB +
                                                           (int64_t)min(m, p.M - 1) * p.do_sM + h_ * p.do_sH);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c * 8 < p.D) {
            o_next[c] = __ldcg(orow + c);
            do_next[c] = __ldcg(grow + c);
          }
      }
    };
    // rowsum(o * dO) in the order of fa_bwd_pre.cu: eight columns one after the other, then pairs
    auto delta_of_next = [&]() {
      float part[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        part[c] = 0.f;
        if (c * 8 < p.D) {
          const uint32_t a[4] = {o_next[ONE_TILE ? c : 0].x, o_next[ONE_TILE ? c : 0].y, o_next[ONE_TILE ? c : 0].z, o_next[ONE_TILE ? c : 0].w};
          const uint32_t g[4] = {do_next[ONE_TILE ? c : 0].x, do_next[ONE_TILE ? c : 0].y, do_next[ONE_TILE ? c : 0].z, do_next[ONE_TILE ? c : 0].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = P2::unpack(a[i]), y = P2::unpack(g[i]);
            part[c] = fmaf(x.x, y.x, part[c]);
            part[c] = fmaf(x.y, y.y, part[c]);
          }
        }
      }
      return ((part[0] + part[4]) + (part[2] + part[6])) + ((part[1] + part[5]) + (part[3] + part[7]));
    };
    // Loop state is kept small on purpose (registers): the running step count gs, the tile
    // counter it, and per tile bh, col0 and the current query block mb; the first query block
    // of a tile is recomputed from col0 where needed.
    uint32_t gs = 0;  // steps done so far, over all tiles
    int bh, nb, i_start, T_steps;
    if (ok && tile_at(0, bh, nb, i_start, T_steps) && T_steps > 0) prefetch(bh, nb * 128 + qt * kCW, i_start);
    // What the last look at the barriers of the coming step saw (nothing yet).  "dV of step -1 has read P" and "dK of step
    // -1 has read dS" hold from the start: a fresh barrier answers the parity of the phase before its first with yes.
    uint32_t ps = 0, pdv = 0, pb = 0;
#pragma unroll 1
    for (int it = 0; ok && tile_at(it, bh, nb, i_start, T_steps); ++it) {
      const int col0 = nb * 128 + qt * kCW;
      if (p.zero_tiles) {
        // sDS becomes the zero tile for the causally skipped part of dbias: the last dbias
        // store of the previous tile must have read it (the last dK product has: its barrier
        // was seen in that tile's epilogue).  Causal completions of st_done: tile `it` owns
        // indices gs+it (zero tiles out) and gs+it+1+t (store of step t).
        if (it >= 1) ok = wait_warp(&st_done, (gs + it - 1) & 1, ctx, kSiteStDone, it);
        if (!ok) break;
        const uint32_t z = sp_row - static_cast<uint32_t>(r) * 128u - (qt * kCW / 64) * kBlk + (L::kDs - L::kP);
        for (int i = tid; i < 2 * kBlk / 16; i += 32 * kRW) sts128(z + i * 16, 0, 0, 0, 0);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&zero_ready);
      }

#pragma unroll 1
      for (int mb = i_start; mb < n_mblk && ok; ++mb, ++gs) {
        const int i0 = p.causal ? min(col0 >> 7, n_mblk) : 0;  // first query block of the tile
        const int t = mb - i0;
        const int m0 = mb * 128;
        if constexpr (ONE_TILE) {
          delta_next = delta_of_next();
          if (qt == 0 && row_ok_next) p.delta_out[(int64_t)bh * p.M + m0 + r] = delta_next;
        }
        BiasRegs<BR> bcur[kNG];
#pragma unroll
        for (int g = 0; g < kNG; ++g) bcur[g] = bnext[g];
        if constexpr (BR == 3) {
          // fp32 bias row of this step: asked for now, used once S has arrived
          const int b_ = bh / p.H, h_ = bh - b_ * p.H;
#pragma unroll
          for (int g = 0; g < kNG; ++g)
            load_bias_row<3>(bcur[g], p.bias, b_ * p.bias_sB + h_ * p.bias_sH + (int64_t)(m0 + r) * p.bias_sM,
                             m0 + r < p.M, col0 + g * 32, p.N, p.bias_vec32 != 0);
        }
        // rows beyond M get -inf / 0, which makes their P and dS zero
        const float neg_lse = row_ok_next ? -lse_next : -INFINITY, delta_r = row_ok_next ? delta_next : 0.f;
        if (!ONE_TILE && mb + 1 < n_mblk) prefetch(bh, col0, mb + 1);
        // ---- P
        ok = wait_warp_polled(ps, &s_full, gs & 1, ctx, kSiteSFull, t);
        if (!ok) break;
        tc_fence_after();
        float pr[kCW];
#pragma unroll
        for (int g = 0; g < kNG; ++g) tmem_ld32(tm_sc + g * 32, reinterpret_cast<uint32_t*>(pr) + g * 32);
        tmem_ld_wait();
        // S now lives in registers: hand its columns back for the next S
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free);
        // P = exp2(S * scale * log2e + bias * log2e - LSE2); rows beyond M have LSE2 = +inf
        // the tile of a bias brought in by TMA: own shared memory, or where this thread's P chunks go
        const uint32_t b_slot = L::kOwnBias ? gs & 1 : 0, b_par = (L::kOwnBias ? gs >> 1 : gs) & 1;
        if constexpr (BIAS == 1) {
          // what does not need the bias is computed while it travels: x = S * scale * log2e - LSE2
          const uint32_t b_row = L::kOwnBias ? sp_row + (L::kBias - L::kP) + b_slot * L::kBiasTile : sp_row;
#pragma unroll
          for (int i = 0; i < kCW; i += 2) {
            const f32x2 x = ffma2(f2(pr[i], pr[i + 1]), f2(p.scale_log2, p.scale_log2), f2(neg_lse, neg_lse));
            pr[i] = f2_lo(x);
            pr[i + 1] = f2_hi(x);
          }
          ok = wait_warp_polled(pb, &bias_full[b_slot], b_par, ctx, kSiteBiasFull, t);
          if (!ok) break;
#pragma unroll
          for (int c = 0; c < kCW / 8; ++c) {
            const uint4 v = lds128(b_row + (((chunk0 + c) ^ (r & 7)) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = P2::unpack(w[e]);
              const int i = c * 8 + e * 2;
              const f32x2 a = ffma2(f2(f.x, f.y), f2(kLog2e, kLog2e), f2(pr[i], pr[i + 1]));
              const f32x2 pe = f2(ex2(f2_lo(a)), ex2(f2_hi(a)));
              pr[i] = f2_lo(pe);
              pr[i + 1] = f2_hi(pe);
            }
          }
        } else {
        BiasRegs<2> mask[kNG];  // of a mask tile: [128 rows][128 bytes]
        if constexpr (BIAS == 2) {
          if constexpr (L::kOwnBias) {
            ok = wait_warp_polled(pb, &bias_full[b_slot], b_par, ctx, kSiteBiasFull, t);
            if (!ok) break;
            const uint32_t m_row = smem_u32(smem + L::kBias) + b_slot * L::kBiasTile + static_cast<uint32_t>(r) * 128u;
#pragma unroll
            for (int c = 0; c < kCW / 16; ++c) {
              const uint4 v = lds128(m_row + (static_cast<uint32_t>((qt * (kCW / 16) + c) ^ (r & 7)) << 4));
              uint32_t* const w = mask[c / 2].w + (c & 1) * 4;
              w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
            }
          } else {
#pragma unroll
            for (int g = 0; g < kNG; ++g)
#pragma unroll
              for (int i = 0; i < 8; ++i) mask[g].w[i] = bcur[g].w[i % (sizeof(bcur[g].w) / 4)];
          }
        }
#pragma unroll
        for (int i = 0; i < kCW; i += 2) {
          f32x2 a = ffma2(f2(pr[i], pr[i + 1]), f2(p.scale_log2, p.scale_log2), f2(neg_lse, neg_lse));
          if (BK == 3)
            a = ffma2(f2(__uint_as_float(bcur[i / 32].w[i % 32]), __uint_as_float(bcur[i / 32].w[i % 32 + 1])), f2(kLog2e, kLog2e), a);
          const f32x2 pe = f2(ex2(f2_lo(a)), ex2(f2_hi(a)));
          if (BK == 2) {
            const uint32_t m2 = mask[i / 32].w[(i % 32) >> 2] >> (8 * (i & 3));
            pr[i] = (m2 & 0xFFu) != 0 ? f2_lo(pe) : 0.f;
            pr[i + 1] = (m2 & 0xFF00u) != 0 ? f2_hi(pe) : 0.f;
          } else {
            pr[i] = f2_lo(pe);
            pr[i + 1] = f2_hi(pe);
          }
        }
        }
        if ((col0 + kCW > p.N) || (p.causal && col0 + kCW - 1 > m0)) {
          int limit = p.N - col0;
          if (p.causal) limit = min(limit, m0 + r - col0 + 1);
#pragma unroll
          for (int i = 0; i < kCW; ++i)
            if (i >= limit) pr[i] = 0.f;
        }
        if (!kBiasInP) {  // (a bias tile lands there after it)
          ok = wait_warp_polled(pdv, &dv_done, (gs - 1) & 1, ctx, kSiteDvDone, t);
          if (!ok) break;
        }
#pragma unroll
        for (int c = 0; c < kCW / 8; ++c)
          sts128(sp_row + (((chunk0 + c) ^ (r & 7)) << 4), P2::pack(pr[c * 8 + 0], pr[c * 8 + 1]),
                 P2::pack(pr[c * 8 + 2], pr[c * 8 + 3]), P2::pack(pr[c * 8 + 4], pr[c * 8 + 5]),
                 P2::pack(pr[c * 8 + 6], pr[c * 8 + 7]));
        // dP, "dK of the previous step has read dS" and "its store has": one combined look, asked for before the fence.
        // sDS may be rewritten once its previous store has read it: with zero tiles completion gs+it of st_done (see
        // above); otherwise completion gs-1 (the store of step gs-1)
        uint32_t pdp, pdk, pst;
        uint64_t* const st_bar = p.store_ds ? &st_done : &dk_done;
        const uint32_t st_par = (p.zero_tiles ? gs + it : gs - 1) & 1;
        mbar_poll3(&dp_full, gs & 1, &dk_done, (gs - 1) & 1, st_bar, st_par, pdp, pdk, pst);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&p_ready);
          if constexpr (L::kOwnBias) mbar_arrive(&bias_empty[b_slot]);  // all that was read from it has gone into P
        }

        // ---- dS
        ok = wait_warp_polled(pdp, &dp_full, gs & 1, ctx, kSiteDpFull, t);
        if (!ok) break;
        tc_fence_after();
        uint32_t dsu[kCW / 2];
        // dP is fetched 16 columns at a time: fewer registers are live at once
#pragma unroll
        for (int hf = 0; hf < kCW / 16; ++hf) {
          uint32_t dp[16];
          tmem_ld16(tm_sc + (kColDp - kColS) + hf * 16, dp);
          tmem_ld_wait();
          if (hf == kCW / 16 - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&dp_free);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = hf * 16 + 2 * i;
            const f32x2 d = fmul2(f2(pr[e], pr[e + 1]),
                                  fadd2(f2(__uint_as_float(dp[2 * i]), __uint_as_float(dp[2 * i + 1])),
                                        f2(-delta_r, -delta_r)));
            dsu[hf * 8 + i] = P2::pack(f2_lo(d), f2_hi(d));
            if (BIAS == 3) {
              dp[2 * i] = __float_as_uint(f2_lo(d));
              dp[2 * i + 1] = __float_as_uint(f2_hi(d));
            }
          }
          if (BIAS == 3 && p.dbias_f32 != nullptr && m0 + r < p.M) {
            // the fp32 bias gradient goes out unrounded, 64 contiguous bytes per thread and fetch
            const int b_ = bh / p.H, h_ = bh - b_ * p.H;
            const int c0 = col0 + hf * 16;
            float* drow = p.dbias_f32 + b_ * p.dbf_sB + h_ * p.dbf_sH + (int64_t)(m0 + r) * p.dbf_sM + c0;
            if (c0 + 16 <= p.N) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint4*>(drow + 4 * k) = make_uint4(dp[4 * k], dp[4 * k + 1], dp[4 * k + 2], dp[4 * k + 3]);
            } else {
#pragma unroll
              for (int k = 0; k < 16; ++k)
                if (c0 + k < p.N) drow[k] = __uint_as_float(dp[k]);
            }
          }
        }
        if (!__all_sync(0xffffffffu, (pdk & pst) != 0)) {
          ok = mbar_wait(&dk_done, (gs - 1) & 1, ctx, kSiteDkDone, t) && mbar_wait(st_bar, st_par, ctx, kSiteStDone, t);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
#pragma unroll
        for (int c = 0; c < kCW / 8; ++c)
          sts128(sp_row + (L::kDs - L::kP) + (((chunk0 + c) ^ (r & 7)) << 4), dsu[c * 4 + 0],
                 dsu[c * 4 + 1], dsu[c * 4 + 2], dsu[c * 4 + 3]);
        // the looks of the next step, of this tile or the next one, are asked for before the fence
        if (L::kOwnBias)
          mbar_poll3(&s_full, (gs + 1) & 1, &dv_done, gs & 1, &bias_full[(gs + 1) & 1], ((gs + 1) >> 1) & 1, ps, pdv, pb);
        else if (kBiasInP)
          mbar_poll2(&s_full, (gs + 1) & 1, &bias_full[0], (gs + 1) & 1, ps, pb);
        else
          mbar_poll2(&s_full, (gs + 1) & 1, &dv_done, gs & 1, ps, pdv);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ds_ready);

        if constexpr (ONE_TILE) {
          // the rows of the next step travel while dQ is formed and stored
          if (mb + 1 < n_mblk) {
            prefetch(bh, col0, mb + 1);
          } else {
            int bh2, nb2, is2, T2;
            if (tile_at(it + 1, bh2, nb2, is2, T2)) prefetch(bh2, nb2 * 128 + qt * kCW, is2);
          }
          ok = wait_warp(&dk_done, gs & 1, ctx, kSiteDkDone, mb);
          if (!ok) break;
          tc_fence_after();
          uint32_t a[32];
          tmem_ld32(tm_sc - qt * kCW + kColDq + qt * 32, a);
          tmem_ld_wait();
          tc_fence_before();
          if (m0 + r < p.M) {
            const int b_ = bh / p.H, h_ = bh - b_ * p.H;
            T* row = static_cast<T*>(p.dq) + b_ * p.dq_sB + (int64_t)(m0 + r) * p.dq_sM + h_ * p.dq_sH;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const int d = qt * 32 + c * 8;
              if (d < p.D) *reinterpret_cast<uint4*>(row + d) = pack8<P2>(a + c * 8, p.sm_scale);
            }
          }
        }
      }
      if (!ok) break;

      // the next tile's first bias / LSE / delta rows travel while this tile's result is stored
      if (!ONE_TILE) {
        int bh2, nb2, is2, T2;
        if (tile_at(it + 1, bh2, nb2, is2, T2) && T2 > 0) prefetch(bh2, nb2 * 128 + qt * kCW, is2);
      }

      // ---- epilogue: dV, dK (rows = keys) -> global
      const int steps_here = n_mblk - (p.causal ? min(col0 >> 7, n_mblk) : 0);
      if (steps_here > 0) {
        ok = wait_warp(&dv_done, (gs - 1) & 1, ctx, kSiteEpilogue, 0);
        if (!ok) break;
      }
      {
        tc_fence_after();
        const int b = bh / p.H, h = bh - b * p.H;
        const int n = (col0 & ~127) + r;
        constexpr int kQD = DP * kCW / 128;  // columns of the head dim this thread stores
        constexpr int kQL = kQD > 32 ? 32 : kQD;
        const int d0 = qt * kQD;
        T* dkrow = reinterpret_cast<T*>(p.dk) + b * p.dk_sB + (int64_t)n * p.dk_sN + h * p.dk_sH;
        T* dvrow = reinterpret_cast<T*>(p.dv) + b * p.dv_sB + (int64_t)n * p.dv_sN + h * p.dv_sH;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          if (which == 1 && steps_here > 0) {  // dV is on its way while the last dK product still runs
            ok = wait_warp(&dk_done, (gs - 1) & 1, ctx, kSiteEpilogue, 1);
            if (!ok) break;
            tc_fence_after();
          }
          T* row = which == 0 ? dvrow : dkrow;
          const uint32_t colbase = which == 0 ? kColDv : kColDk;
          const float mul = which == 0 ? 1.0f : p.sm_scale;
          uint32_t a[kQD];
          if (steps_here > 0) {
#pragma unroll
            for (int c = 0; c < kQD; c += kQL) tmem_ld_cols<kQL>(tm_sc - qt * kCW + colbase + d0 + c, a + c);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < kQD; ++i) a[i] = 0;
          }
          if (n < p.N) {
            if (p.dkv_vec32 && d0 + kQD <= p.D) {
              // whole 32-byte sectors per store: half as many transactions as 16-byte stores for
              // these row-strided writes
#pragma unroll
              for (int c = 0; c < kQD / 16; ++c) {
                const uint4 lo = pack8<P2>(a + c * 16, mul), hi = pack8<P2>(a + c * 16 + 8, mul);
                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(row + d0 + c * 16),
                             "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
                             : "memory");
              }
            } else {
#pragma unroll
              for (int c = 0; c < kQD / 8; ++c) {
                const int d = d0 + c * 8;
                if (d < p.D) *reinterpret_cast<uint4*>(row + d) = pack8<P2>(a + c * 8, mul);
              }
            }
          }
        }
        // the accumulators are in registers: the next tile's first products may overwrite them
        tc_fence_before();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kRW + 1) tmem_dealloc(tmem, kTmemCols);
}

template <int DP, typename T, int BIAS, bool LONGEST_FIRST, bool ONE_TILE = false>
int launch_inst(const DkdvParams& kp, dim3 grid, cudaStream_t stream) {
  using L = DkdvSmem<DP, BIAS>;
  auto kern = dkdv_kernel<DP, T, BIAS, LONGEST_FIRST, ONE_TILE>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamic) !=
        cudaSuccess)
      return FA_ERR_CUDA;
    configured[dev] = true;
  }
  return launch_overlapped(kern, grid, kThreads, L::kDynamic, stream, kp);
}

template <int DP, typename T, bool LONGEST_FIRST>
int launch_bias(const DkdvParams& kp, int bias_kind, dim3 grid, cudaStream_t stream) {
  switch (bias_kind) {
    case FA_BIAS_NONE: return launch_inst<DP, T, 0, LONGEST_FIRST>(kp, grid, stream);
    case FA_BIAS_SAME: return launch_inst<DP, T, 1, LONGEST_FIRST>(kp, grid, stream);
    case FA_BIAS_BOOL: return launch_inst<DP, T, 2, LONGEST_FIRST>(kp, grid, stream);
    case FA_BIAS_F32: return launch_inst<DP, T, 3, LONGEST_FIRST>(kp, grid, stream);
    default: return FA_ERR_UNSUPPORTED;
  }
}
template <typename T>
int launch_one_tile(const DkdvParams& kp, int bias_kind, dim3 grid, cudaStream_t stream) {
  switch (bias_kind) {
    case FA_BIAS_NONE: return launch_inst<64, T, 0, false, true>(kp, grid, stream);
    case FA_BIAS_SAME: return launch_inst<64, T, 1, false, true>(kp, grid, stream);
    case FA_BIAS_BOOL: return launch_inst<64, T, 2, false, true>(kp, grid, stream);
    case FA_BIAS_F32: return launch_inst<64, T, 3, false, true>(kp, grid, stream);
    default: return FA_ERR_UNSUPPORTED;
  }
}
template <bool LONGEST_FIRST>
int launch_dim(const DkdvParams& kp, int dtype, int bias_kind, dim3 grid, cudaStream_t stream) {
  const bool dp64 = padded_head_dim(kp.D) == 64;
  if (dtype == FA_BF16)
    return dp64 ? launch_bias<64, __nv_bfloat16, LONGEST_FIRST>(kp, bias_kind, grid, stream)
                : launch_bias<128, __nv_bfloat16, LONGEST_FIRST>(kp, bias_kind, grid, stream);
  return dp64 ? launch_bias<64, __half, LONGEST_FIRST>(kp, bias_kind, grid, stream)
              : launch_bias<128, __half, LONGEST_FIRST>(kp, bias_kind, grid, stream);
}

// Work of key block `nb` of a causal problem, in quarters of a step: four a step, six for the tile's boundary and `zeros`
// for each zero tile that a 16-bit bias gradient gets above the diagonal.  A block that no query sees only stores zeros.
int tile_work(int nb, int n_mblk, int zeros) {
  const int steps = n_mblk - nb;
  return steps > 0 ? 4 * steps + 6 + zeros * nb : 3 + zeros * n_mblk;
}

}  // namespace

int dkdv_pair_work(const fa_params& p) {
  const int n_mblk = (p.M + 127) / 128;
  return tile_work(0, n_mblk, 0) + tile_work((p.N + 127) / 128 - 1, n_mblk, 0);
}

// Causal pairs of a heavy and a light tile leave CTAs idle in their last turn, with an odd number of key blocks also
// before it, and one pair a CTA leaves half of the CTAs without one.  Longest first the tiles spread better, but a head's
// tiles no longer run side by side: only up to four a CTA, so that all operands stay in L2 without an order by head.
// The longest CTA of both orders decides, with 3 % for the pairs, and 6 % where a bias is read in more than two rows of
// tiles (its sectors are shared by neighbouring key blocks).
// Measured over 1382 calls (whole backward; D 64 and 128, four kinds of bias, 512 to 8192 keys, M = N and not): of the 1132
// taken 10 lose more than 1.5 % (at most 5 %, 25 us calls of 1024 x 2048), of those left to the pairs 7 would have gained as
// much (at most 2.4 %); the mean gain over all is 8.9 %.  Pairs / longest first, us (estimate, measured):
//   S1024 D64: H45 63.9 / 51.0 (1.45, 1.25)   H64 71.9 / 69.6 (1.09, 1.03)   H72 74.6 / 77.1 (1.00, 0.97: pairs)
//   the same, 16-bit bias, H64: 91.4 / 91.3 (1.06, 1.00)   S1000, 16-bit bias, H60: 95.5 / 98.8 (1.06, 0.97: pairs)
//   S1032 D64 H22, nine key blocks: 52.2 / 41.4 (1.62, 1.26)   S4096 D128 H9: 129.8 / 128.3 (1.00, 1.01: pairs)
//   S8192 D128: H2, 16-bit bias 271 / 235 (1.28, 1.15)   H3, fp32 bias 473 / 485 (1.04, 0.98)
DkdvPlan plan_dkdv(const fa_params& p, int n_bh, int sms, bool writes_zeros) {
  const int n_mblk = (p.M + 127) / 128, n_nblk = (p.N + 127) / 128;
  const int64_t all = static_cast<int64_t>(n_nblk) * n_bh;
  if (!p.causal || all > 4 * sms) return {false, 0};
  const int n = static_cast<int>(all), zeros = writes_zeros ? 1 : 0;
  const CausalSpans span = causal_spans(n, n_bh, n_nblk, sms, [&](int nb) { return tile_work(nb, n_mblk, zeros); });
  const int margin = p.bias_kind != FA_BIAS_NONE && n > 2 * sms ? 106 : 103;
  const bool longest_first = 100 * static_cast<int64_t>(span.pairs) >= margin * static_cast<int64_t>(span.longest_first);
  return {longest_first, longest_first ? span.longest_first : span.pairs};
}

// One tile of keys and at most two blocks of queries: dQ joins the chain of a step, which a head walks alone (at B1 H8 M4096
// N128 the streamed dQ kernel has 256 CTAs, this one 8).  Up to two heads a CTA the launches are what a pass waits for; with
// more, three kernels that overlap their tiles are faster, except with an fp32 bias, whose dS would go to scratch and back.
// Training pass, us, three launches / one: B2 S128 H4 D64, 16-bit trained bias 79.9 / 74.0; B4 H16 S128 causal 68.0 / 62.1; B16
// H12 200 x 77, padding mask 76.5 / 69.9; B64 H3 S81 D16, trained table 100.4 / 95.8; fp32 trained bias B8 H4 256 x 128 74.4 / 68.4,
// B500 H8 128 x 100 577 / 536; left to three: trained table B256 H6 S100 D32 143 / 159, B600 H4 S128 D64 210 / 277.
bool one_tile_takes(const fa_params& p) {
  return p.N <= 128 && p.M <= 256 && p.D <= 64 && !small_takes(p.M, p.N, p.D) &&
         (p.bias_kind == FA_BIAS_F32 || p.B * p.H <= 2 * persistent_grid(1 << 30));
}

namespace {

int launch_dkdv(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab, bool one_tile) {
  DkdvParams kp;
  int r = make_tmap_bshd(&kp.map_q, p.q, p.B, p.M, p.H, p.D, p.q_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_k, p.k, p.B, p.N, p.H, p.D, p.k_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_v, p.v, p.B, p.N, p.H, p.D, p.v_stride, 128);
  if (r) return r;
  r = make_tmap_bshd(&kp.map_do, p.d_o, p.B, p.M, p.H, p.D, p.do_stride, 128);
  if (r) return r;
  const bool f32 = p.bias_kind == FA_BIAS_F32;
  kp.ds_flat = slab != nullptr;
  kp.bh0 = slab ? slab->bh0 : 0;
  // (one tile of keys: nothing reads dS back, but a caller that gives a ds16 finds it there all the same)
  kp.store_ds = slab || (f32 && (!one_tile || p.ds16)) || (!f32 && p.write_dbias);
  kp.zero_tiles = !f32 && p.write_dbias && p.causal;
  kp.dbias_f32 = nullptr;
  kp.dbf_sB = kp.dbf_sH = kp.dbf_sM = 0;
  if (slab) {
    r = make_tmap_slab(&kp.map_dbias, *slab, p.M, p.N);
    if (r) return r;
  } else if (kp.store_ds) {
    // the 16-bit dS tiles: the bias gradient itself, or (fp32 bias) the scratch the dQ stage reads
    const void* dst = f32 ? p.ds16 : p.dbias;
    const int64_t* dst_stride = f32 ? p.ds16_stride : p.dbias_stride;
    if (!dst) return FA_ERR_NULL;
    int bm, hm;
    r = make_tmap_bhmn(&kp.map_dbias, dst, 2, p.B, p.H, p.M, p.N, dst_stride, 64, 128, &bm, &hm);
    if (r) return r;
    if (!bm || !hm) return FA_ERR_ALIGN;  // must be a real (B,H,M,N) tensor
  } else {
    kp.map_dbias = kp.map_q;
  }
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
  auto al32 = [](const void* ptr, const int64_t s[3]) {
    return reinterpret_cast<uintptr_t>(ptr) % 32 == 0 && s[0] % 16 == 0 && s[1] % 16 == 0 && s[2] % 16 == 0;
  };
  kp.dkv_vec32 = al32(p.dk, p.dk_stride) && al32(p.dv, p.dv_stride);
  kp.bias_b_mul = kp.bias_h_mul = 0;
  kp.map_bias = kp.map_q;
  if (p.bias_kind == FA_BIAS_SAME) {
    r = make_tmap_bhmn(&kp.map_bias, p.bias, 2, p.B, p.H, p.M, p.N, p.bias_stride, 64, 128,
                       &kp.bias_b_mul, &kp.bias_h_mul);
    if (r) return r;
  } else if (p.bias_kind == FA_BIAS_BOOL) {
    r = make_tmap_bhmn(&kp.map_bias, p.bias, 1, p.B, p.H, p.M, p.N, p.bias_stride, 128, 128,
                       &kp.bias_b_mul, &kp.bias_h_mul);
    if (r) return r;
  } else if (f32) {
    r = make_tmap_bhmn(&kp.map_bias, p.bias, 4, p.B, p.H, p.M, p.N, p.bias_stride, 32, 128,
                       &kp.bias_b_mul, &kp.bias_h_mul);
    if (r) return r;
  }
  if (p.bias_kind != FA_BIAS_NONE) {
    const int eb = p.bias_kind == FA_BIAS_BOOL ? 1 : (f32 ? 4 : 2);
    if (reinterpret_cast<uintptr_t>(p.bias) % 16 != 0 || (p.bias_stride[0] * eb) % 16 ||
        (p.bias_stride[1] * eb) % 16 || (p.bias_stride[2] * eb) % 16)
      return FA_ERR_ALIGN;
  }
  kp.bias = p.bias;
  kp.dk = p.dk;
  kp.dv = p.dv;
  kp.lse = p.lse;
  kp.delta = p.delta;
  kp.status = status;
  kp.bias_sB = p.bias_stride[0];
  kp.bias_sH = p.bias_stride[1];
  kp.bias_sM = p.bias_stride[2];
  kp.dk_sB = p.dk_stride[0];
  kp.dk_sN = p.dk_stride[1];
  kp.dk_sH = p.dk_stride[2];
  kp.dv_sB = p.dv_stride[0];
  kp.dv_sN = p.dv_stride[1];
  kp.dv_sH = p.dv_stride[2];
  kp.H = p.H;
  kp.M = p.M;
  kp.N = p.N;
  kp.D = p.D;
  kp.causal = p.causal ? 1 : 0;
  {
    const int eb = p.bias_kind == FA_BIAS_BOOL ? 1 : (f32 ? 4 : 2);
    kp.bias_vec32 = p.bias_kind != FA_BIAS_NONE && reinterpret_cast<uintptr_t>(p.bias) % 32 == 0 &&
                    (p.bias_stride[0] * eb) % 32 == 0 && (p.bias_stride[1] * eb) % 32 == 0 &&
                    (p.bias_stride[2] * eb) % 32 == 0;
  }
  kp.scale_log2 = p.sm_scale * kLog2e;
  kp.sm_scale = p.sm_scale;
  kp.n_nblk = (p.N + 127) / 128;
  kp.n_bh = slab ? slab->n_bh : p.B * p.H;
  kp.n_tiles = kp.n_nblk * kp.n_bh;
  const int sms = persistent_grid(1 << 30);
  if (one_tile) {
    if (bad(p.o, p.o_stride) || bad(p.d_o, p.do_stride) || bad(p.dq, p.dq_stride)) return FA_ERR_ALIGN;
    kp.o = p.o, kp.d_o = p.d_o, kp.dq = p.dq, kp.delta_out = p.delta;
    kp.o_sB = p.o_stride[0], kp.o_sM = p.o_stride[1], kp.o_sH = p.o_stride[2];
    kp.do_sB = p.do_stride[0], kp.do_sM = p.do_stride[1], kp.do_sH = p.do_stride[2];
    kp.dq_sB = p.dq_stride[0], kp.dq_sM = p.dq_stride[1], kp.dq_sH = p.dq_stride[2];
    const dim3 grid(kp.n_tiles < sms ? kp.n_tiles : sms);
    return p.dtype == FA_BF16 ? launch_one_tile<__nv_bfloat16>(kp, p.bias_kind, grid, stream)
                              : launch_one_tile<__half>(kp, p.bias_kind, grid, stream);
  }
  const bool longest_first = plan_dkdv(p, kp.n_bh, sms, kp.zero_tiles != 0).longest_first;
  const int units = p.causal && !longest_first ? (kp.n_tiles + 1) / 2 : kp.n_tiles;
  const dim3 grid(units < sms ? units : sms);
  return longest_first ? launch_dim<true>(kp, p.dtype, p.bias_kind, grid, stream)
                       : launch_dim<false>(kp, p.dtype, p.bias_kind, grid, stream);
}

}  // namespace

int launch_bwd_dkdv(const fa_params& p, cudaStream_t stream, int* status, const DsSlab* slab) {
  return p.D == 256 ? launch_bwd_dkdv_d256(p, stream, status, slab) : launch_dkdv(p, stream, status, slab, false);
}

int launch_bwd_one_tile(const fa_params& p, cudaStream_t stream, int* status) {
  return launch_dkdv(p, stream, status, nullptr, true);
}

}  // namespace fa
