// The bf16 GEMM of gemm_bf16.cu for long steps, by pairs of CTAs (tcgen05 cta_group::2).  Included there, behind the LoRA pieces it shares.
//
// A pair takes a tile of 256 output features x up to 256 tokens: each CTA loads 128 rows of the weights and half of the tokens, 32 KB a stage
// where one CTA on its own tile of 128 x 256 takes 48, and reads half the token operand from its shared memory per MMA: what a single CTA
// moves in and out of shared memory per product is the limit of gemm_bf16_tcgen05_kernel at these sizes (192 of about 128 B per cycle asked for).
// 4001 rows, 28672 x 4096: 703 -> 630 to 680 us with the clock, the tensor pipe 90 % active at the 1.5 GHz that the power limit leaves.  Operands carry
// no eviction hints: the pairs of a wave share weight tiles and token tiles through L2 (weights evicted early cost 2 to 3 % of a pass).
// Rank 0's MMA thread issues for both; a stage is full when the loads of both CTAs have arrived at rank 0's barrier, and its commits
// tell both that a stage is free or an accumulator complete.  Whole tiles and the stream-K remainder as there, each CTA with its half of a tile's
// partial sums.  LoRA as there: shrink on the epilogue warps of all CTAs during the first K loop, expand by MMAs into the
// accumulators, whose columns come in steps of 32 here (an entry's window: 64 rows, 32-aligned); each CTA brings its features' B_cat and half of the
// window's rows.  One row of ranks serves both CTAs, so parts must begin at multiples of 256.
#pragma once

#include "pair.cuh"

namespace lx {

constexpr int kPairStages = 6;
constexpr int kPairUnits = 6;                         // expand units that share a stage
constexpr int kPairImgBytes = 32 * 32;                // half of a window's rows, 16 ranks
struct PairHeader {
  LoraUnit units[kPairUnits];
  int nu, last, pad_[2];
};
template <bool LORA>
struct PairSmem {
  static constexpr int kABytes = kBM * kBK * 2, kBBytes = kBM * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static_assert(kPairUnits * (kLoraBTileBytes + kPairImgBytes) + (int)sizeof(PairHeader) <= kStageBytes, "an expand stage fits");
  static constexpr int kBarrierBytes = 256;
  static constexpr int kEntBytes = LORA ? kLoraMaxEntries * (int)sizeof(LoraEnt) + kLoraListCap * 32 + (kLoraMaxEntries + 8) * 2 : 0;
  static constexpr int kEpiBytes = 4 * 32 * 32 * 2;
  static constexpr int kTotal = kPairStages * kStageBytes + kBarrierBytes + kEntBytes + kEpiBytes + 1024;
  static_assert(kTotal <= 227 * 1024, "shared memory of one CTA");
};

using PairIter = GemmWorkIter<256>;
constexpr double kPairFillBytesPerNs = 95.0, kPairSumBytesPerNs = 8.0;

template <bool LORA>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_img,
                 const __grid_constant__ LoraBMaps bmaps, const GemmParams p) {
  using S = PairSmem<LORA>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kPairStages * S::kStageBytes);      // (rank 0's are used)
  uint64_t* empty_bar = full_bar + kPairStages;
  uint64_t* tmem_full = empty_bar + kPairStages;
  uint64_t* tmem_empty = tmem_full + 2;                                                       // (rank 0's are used)
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
  int* n_live = reinterpret_cast<int*>(tmem_base_slot + 3);
  LoraEnt* ents = reinterpret_cast<LoraEnt*>(smem + kPairStages * S::kStageBytes + S::kBarrierBytes);
  LoraUnit* ulist = reinterpret_cast<LoraUnit*>(ents + kLoraMaxEntries);
  unsigned short* gstart = reinterpret_cast<unsigned short*>(ulist + kLoraListCap);
  __nv_bfloat16* epi_stage = reinterpret_cast<__nv_bfloat16*>(smem + kPairStages * S::kStageBytes + S::kBarrierBytes + S::kEntBytes);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  const int tiles_a = (p.a_rows + 2 * kBM - 1) / (2 * kBM), tiles_b = (p.b_rows + p.bn - 1) / p.bn;
  const int num_tiles = tiles_a * tiles_b;
  const int kblocks = (p.K + kBK - 1) / kBK;
  const int half = p.bn >> 1;                          // tokens that this CTA loads
  const bool lora = LORA && p.lora_tiles != nullptr;
  int pre_tb = -1, pre_n = 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tmem_full[s], 1); mbar_init(&tmem_empty[s], 8); }
    *abort_flag = 0;
    *n_live = LORA ? p.lora_num_tiles : 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) pair_tmem_alloc(tmem_base_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                      // both CTAs' barriers and columns are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;
  if constexpr (LORA) {
    if (lora) {
      if (!p.lora_tables_const) pdl_wait();
      load_lora_entries(p, ents, n_live);
      __syncthreads();
      if (warp == 2) lora_unit_prefix(p, ents, gstart);
      PairIter it0(p, num_tiles, kblocks, pairs, pair);
      GemmWork w0;
      if (warp == 0 && it0.next(w0) && w0.kb0 == 0) {
        const int ta0 = w0.tile / tiles_b, tb0 = w0.tile % tiles_b;
        const int n0 = lora_prebuild_units<kLoraPairWin>(p, ents, *n_live, tb0 * p.bn, tb0 * p.bn + p.bn, ulist);
        if (n0 >= 0) { pre_tb = tb0; pre_n = n0; }
        if (n0 > 0) lora_prefetch_b(p, ulist, n0, 2 * ta0 + (int)rank);
      }
      __syncthreads();
    }
  }
  // (see gemm_bf16_tcgen05_kernel: constant weights of the first stages, ahead of the wait)
  int preloaded = 0;
  if (threadIdx.x == 0 && p.w_preload) {
    PairIter it0(p, num_tiles, kblocks, pairs, pair);
    GemmWork w0;
    if (it0.next(w0)) {
      preloaded = min(kPairStages, w0.kb1 - w0.kb0);
      for (int s = 0; s < preloaded; ++s) {
        if (rank == 0) mbar_expect_tx(&full_bar[s], 2u * (uint32_t)(S::kABytes + half * kBK * 2));
        pair_load_2d(tiles + s * S::kStageBytes, &tmap_a, pair_map(&full_bar[s], 0), (w0.kb0 + s) * kBK, (2 * (w0.tile / tiles_b) + (int)rank) * kBM);
      }
    }
  }
  pdl_wait();

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int list_tb = pre_tb, list_n = pre_n;
    bool first_tile = pre_tb >= 0, shrink_seen = false;
    PairIter it(p, num_tiles, kblocks, pairs, pair);
    GemmWork w;
    while (it.next(w)) {
      const int tile = w.tile, ta = tile / tiles_b, tb = tile % tiles_b;
      const int i0 = (2 * ta + (int)rank) * kBM, j0 = tb * p.bn, jlim = j0 + p.bn;
      if constexpr (LORA) {
        if (lora && w.kb0 == 0) {
          if (list_tb != tb) {
            const int n0 = lora_prebuild_units<kLoraPairWin>(p, ents, *n_live, j0, jlim, ulist);
            list_tb = n0 >= 0 ? tb : -1;
            list_n = n0 >= 0 ? n0 : 0;
          }
          if (list_tb == tb && list_n > 0 && !first_tile) lora_prefetch_b(p, ulist, list_n, 2 * ta + (int)rank);
          first_tile = false;
        }
      }
      if (lane == 0 && ok) {
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          const bool have = preloaded > 0;
          if (have) {
            --preloaded;
          } else if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
            report_status(p.status, kTimeoutEmptyBarrier, tile);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = tiles + stage * S::kStageBytes;
          const uint32_t bar = pair_map(&full_bar[stage], 0);
          if (rank == 0 && !have) mbar_expect_tx(&full_bar[stage], 2u * (uint32_t)(S::kABytes + half * kBK * 2));
          if (!have) pair_load_2d(sa, &tmap_a, bar, kb * kBK, i0);
          pair_load_2d(sa + S::kABytes, &tmap_b, bar, kb * kBK, j0 + (int)rank * half);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
      }
      if constexpr (LORA) {
        if (lora && w.kb0 == 0) {
          __syncwarp();
          stage = __shfl_sync(0xffffffffu, stage, 0);
          phase = __shfl_sync(0xffffffffu, phase, 0);
          ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
          const int pt = min(p.lora_nparts - 1, i0 < p.lora_n0 ? 0 : (i0 < p.lora_n1 ? 1 : 2));
          const long long img_part = (long long)pt * 4 * p.lora_num_tiles;
          if (ok && !shrink_seen) {
            if (lane == 0) {
              if (!wait_flag(&p.lora_sync[1], (int)gridDim.x, abort_flag)) {
                report_status(p.status, kTimeoutSplitK, tile);
                *abort_flag = 1;
              }
            }
            __syncwarp();
            ok = (*abort_flag == 0);
            fence_proxy_async_all();       // the images were written with ordinary stores; the loads below are the async proxy's
            shrink_seen = true;
          }
          auto send_stage = [&](int base, int nu, bool last) -> bool {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
              if (lane == 0) {
                report_status(p.status, kTimeoutEmptyBarrier, tile);
                *abort_flag = 1;
              }
              return false;
            }
            uint8_t* sa = tiles + stage * S::kStageBytes;
            PairHeader* hdr = reinterpret_cast<PairHeader*>(sa + kPairUnits * (kLoraBTileBytes + kPairImgBytes));
            LoraUnit q{};
            if (lane < nu) q = ulist[base + lane];
            const int rows = lane < nu ? (q.c1 - q.c0) >> 1 : 0;                  // of the window, in each CTA: 16 or 32
            const int bytes = __reduce_add_sync(0xffffffffu, lane < nu ? kLoraBTileBytes + rows * 32 : 0);
            const uint32_t bar = pair_map(&full_bar[stage], 0);
            if (rank == 0) {
              if (lane < nu) hdr->units[lane] = q;
              if (lane == 0) { hdr->nu = nu; hdr->last = last ? 1 : 0; }
              fence_proxy_async_smem();          // the stage's bytes are written by bulk copies at other times
              __syncwarp();
              if (lane == 0) mbar_expect_tx(&full_bar[stage], 2u * (uint32_t)bytes);
            }
            __syncwarp();
            if (lane < nu) {
              pair_load_3d(sa + lane * kLoraBTileBytes, &bmaps.m[q.rclass], bar, (q.img & 3) * 16, i0, q.boff);
              const int row = (int)(img_part + (long long)(q.img & 3) * p.lora_num_tiles + (q.img >> 2)) * kLoraPairWin + (q.c0 - q.w0) + (int)rank * rows;
              uint8_t* dst = sa + kPairUnits * kLoraBTileBytes + lane * kPairImgBytes;
              for (int h = 0; h < rows; h += 16) pair_load_2d(dst + h * 32, &tmap_img, bar, 0, row + h);
            }
            if (++stage == kPairStages) { stage = 0; phase ^= 1; }
            return true;
          };
          auto send_run = [&](int n, bool closes) {
            if (n == 0 && closes) ok = send_stage(0, 0, true);
            for (int base = 0; ok && base < n; base += kPairUnits) ok = send_stage(base, min(kPairUnits, n - base), closes && base + kPairUnits >= n);
          };
          if (!ok) {
          } else if (list_tb == tb) {
            send_run(list_n, true);
          } else {
            // more units than the list holds: built and sent in pieces
            int n = 0;
            bool ended = false;
            for (int lt0 = lora_first_entry<kLoraPairWin>(ents, *n_live, j0); ok; lt0 += 32) {
              bool last = true;
              if (lt0 < p.lora_num_tiles) {
                n = lora_build_units<kLoraPairWin>(p, ents, lt0, j0, jlim, ulist, n, ended);
                last = ended || lt0 + 32 >= p.lora_num_tiles;
                if (n < 128 && !last) continue;
              }
              send_run(n, last);
              if (last) break;
              n = 0;
            }
          }
        }
      }
    }
    __syncwarp();
    if (p.overlap) pdl_launch_dependents();      // the last loads of this CTA are on their way: the next kernel's blocks may be set up
  } else if (warp == 1) {
    if (rank == 0 && lane == 0) {
      const uint32_t idesc = make_idesc(2 * kBM, (uint32_t)p.bn, kFmtBF16, kFmtBF16);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase[2] = {0, 0};
      bool ok = true;
      PairIter it(p, num_tiles, kblocks, pairs, pair);
      GemmWork w;
      while (ok && it.next(w)) {
        const int tile = w.tile;
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * 256);
        if (!pair_wait(&tmem_empty[acc], acc_phase[acc] ^ 1, abort_flag)) {
          report_status(p.status, kTimeoutTmemEmpty, tile);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
            report_status(p.status, kTimeoutFullBarrier, tile);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * S::kStageBytes);
          const uint64_t da = make_desc_k_sw128(sa), db = make_desc_k_sw128(sa + S::kABytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) pair_mma(tmem_d, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, (kb > w.kb0 || k > 0) ? 1u : 0u);
          pair_commit(&empty_bar[stage]);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
        if constexpr (LORA) {
          bool more = lora && ok && w.kb0 == 0;
          while (more) {
            if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
              report_status(p.status, kTimeoutFullBarrier, tile);
              *abort_flag = 1;
              ok = false;
              break;
            }
            tc_fence_after();
            uint8_t* sp = tiles + stage * S::kStageBytes;
            const PairHeader* hdr = reinterpret_cast<const PairHeader*>(sp + kPairUnits * (kLoraBTileBytes + kPairImgBytes));
            const uint32_t sa = smem_u32(sp);
            const int nu = min(hdr->nu, kPairUnits), j0 = tile % tiles_b * p.bn;
            more = hdr->last == 0;
            for (int u = 0; u < nu; ++u) {
              const LoraUnit q = hdr->units[u];
              pair_mma(tmem_d + (uint32_t)(q.c0 - j0), make_desc_k_sw32(sa + (uint32_t)(u * kLoraBTileBytes)),
                       make_desc_k_sw32(sa + (uint32_t)(kPairUnits * kLoraBTileBytes + u * kPairImgBytes)),
                       make_idesc(2 * kBM, (uint32_t)(q.c1 - q.c0), kFmtBF16, kFmtBF16), 1u);
            }
            pair_commit(&empty_bar[stage]);
            if (++stage == kPairStages) { stage = 0; phase ^= 1; }
          }
        }
        if (ok) pair_commit(&tmem_full[acc]);
        acc_phase[acc] ^= 1;
        acc ^= 1;
      }
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;
    int acc = 0;
    uint32_t acc_phase[2] = {0, 0};
    if constexpr (LORA) {
      if (lora) lora_shrink_units<kLoraPairWin>(p, ents, gstart, reinterpret_cast<float*>(epi_stage), warp - 2, lane);
    }
    const bool turn = p.ldo_a == 1 && (p.ldo_b & 7) == 0 && (p.a_rows & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
    PendingTile pending[2];
    int n_pending = 0;
    bool alive = true;
    PairIter it(p, num_tiles, kblocks, pairs, pair);
    GemmWork w;
    while (it.next(w)) {
      const int tile = w.tile, ta = tile / tiles_b, tb = tile % tiles_b;
      if (!mbar_wait(&tmem_full[acc], acc_phase[acc], abort_flag)) {
        report_status(p.status, kTimeoutTmemFull, tile);
        *abort_flag = 1;
        alive = false;
        break;
      }
      tc_fence_after();
      acc_phase[acc] ^= 1;
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * 256);
      if (w.nparts > 0) {
        // part of a tile's K: both CTAs park their half, [column][128 features] fp32, and count in; the sums follow behind the last unit
        constexpr long long kPart = 256ll * kBM;
        float* wsp = p.ws + 2 * w.part_off + rank * kPart + quad * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < p.bn; c += 32) {
          if (tb * p.bn + c >= p.b_rows) break;
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c, r);
          tc_wait_ld();
#pragma unroll
          for (int q = 0; q < 32; ++q) __stcg(wsp + (long long)(c + q) * kBM, __uint_as_float(r[q]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) pair_arrive(pair_map(&tmem_empty[acc], 0));
        __threadfence();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        const int counter = 2 * w.counter + (int)rank;
        if (threadIdx.x == 64) atomicAdd(&p.counters[counter], 1);
        if (n_pending < 2)
          pending[n_pending++] = PendingTile{(2 * ta + (int)rank) * kBM, tb, counter, w.nparts, w.part_idx, 2 * w.red_first + rank * kPart,
                                             2 * w.red_base + rank * kPart, 2 * w.red_stride};
        acc ^= 1;
        continue;
      }
      const int f0 = (2 * ta + (int)rank) * kBM + quad * 32, i = f0 + lane;
      const int j0 = tb * p.bn, jend = min(p.b_rows, j0 + p.bn);
      const float bias_i = (p.bias != nullptr && i < p.a_rows) ? __bfloat162float(p.bias[i]) : 0.f;
      __nv_bfloat16* st = epi_stage + quad * (32 * 32);
      const int fbase = f0 + (lane & 3) * 8;
#pragma unroll 1
      for (int c = 0; c < p.bn; c += 32) {
        if (j0 + c >= jend) break;
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + c, r);
        tc_wait_ld();
        if (turn) {
          // a thread holds one feature of 32 tokens; the warp turns its block around and stores eight features of a token per lane
#pragma unroll
          for (int q = 0; q < 32; ++q) st[q * 32 + lane] = __float2bfloat16(__uint_as_float(r[q]) * p.out_scale + bias_i);
          __syncwarp();
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int tq = h * 8 + (lane >> 2), t = j0 + c + tq;
            if (t < jend && fbase < p.a_rows)
              *reinterpret_cast<uint4*>(p.out + (long long)t * p.ldo_b + fbase) = *reinterpret_cast<const uint4*>(st + tq * 32 + (lane & 3) * 8);
          }
          __syncwarp();
        } else if (i < p.a_rows) {
#pragma unroll
          for (int q = 0; q < 32; ++q)
            if (j0 + c + q < jend)
              p.out[(long long)i * p.ldo_a + (long long)(j0 + c + q) * p.ldo_b] = __float2bfloat16(__uint_as_float(r[q]) * p.out_scale + bias_i);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) pair_arrive(pair_map(&tmem_empty[acc], 0));
      acc ^= 1;
    }
    for (int i = 0; alive && i < n_pending; ++i) alive = gemm_sum_share(p, pending[i], abort_flag);
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();                                      // nothing of this pair is on its way to a CTA that has left
  if (warp == 1) {
    tc_fence_after();
    pair_tmem_dealloc(tmem_base, 512);
  }
  if constexpr (LORA) {
    if (lora && threadIdx.x == 0) {
      __threadfence();
      const int prev = atomicAdd(&p.lora_sync[0], 1);
      if (prev == (int)gridDim.x - 1) {
        p.lora_sync[0] = 0;
        p.lora_sync[1] = 0;
        __threadfence();
      }
    }
  }
}

// (the wait for the shrink counts on the pairs running at the same time)
template <bool LORA>
static int pair_capacity() {
  static int known[64] = {0};
  return pair_capacity_of(gemm_pair_kernel<LORA>, kGemmThreads, PairSmem<LORA>::kTotal, known);
}

struct PairPlan {
  int bn, dp_tiles, sk_pairs, grid;      // token tile (0: no plan); whole tiles; pairs that share the K of the others; pairs
  double cost;                           // ns
};
// The token tile, a multiple of 32, that costs least.  A k-block takes as long as its operands take to come in from L2, 128 rows of weights and
// half its tokens per CTA (their MMAs need less than that); a tile has a start, and the sums of a shared one their trips through L2.
// (ws_bytes: scratch of the sums; without it all tiles are whole.)
static PairPlan pair_plan(int T, int N, int K, int pairs, long long ws_bytes) {
  PairPlan best{};
  best.cost = 1e30;
  const int kblocks = (K + kBK - 1) / kBK, tiles_a = (N + 255) / 256;
  const int top = (T + 31) / 32 * 32 < 256 ? (T + 31) / 32 * 32 : 256;
  for (int bn = top; bn >= 32; bn -= 32) {
    const long long tiles = (long long)tiles_a * ((T + bn - 1) / bn);
    const double block = (kBM + bn / 2) * 128.0 / kPairFillBytesPerNs, start = kTileFixedNs;
    const long long full = tiles / pairs, rest = tiles - full * pairs;
    PairPlan w{bn, (int)tiles, 0, (int)(tiles < pairs ? tiles : pairs), (double)(full + (rest ? 1 : 0)) * (kblocks * block + start)};
    if (w.cost < best.cost) best = w;
    if (rest == 0) continue;
    long long sk = pairs;
    if (sk > rest * kblocks / 2) sk = rest * kblocks / 2;
    if (sk > 15 * rest) sk = 15 * rest;
    if (sk <= rest || sk * 4 * 256 * kBM * 4 > ws_bytes) continue;
    const double parts = (double)kBM * bn * 4.0 / kPairSumBytesPerNs + 2500.0;
    PairPlan q{bn, (int)(full * pairs), (int)sk, full ? pairs : (int)sk, full * (kblocks * block + start) + (double)rest * kblocks / sk * block + start + parts};
    if (q.cost < best.cost) best = q;
  }
  return best;
}

// The same, with token tile 0 where single CTAs (a plan of `single_cost`) are as quick.  Both costs leave out what every launch has, and pairs have more
// of it (two barriers of the cluster, columns allocated for both): 4 us and 15 % of the pairs' cost is where they are worth it over 2960 shapes of 193
// to 4001 rows, 256 to 28672 features, K 128 to 14336.  Where the rule takes pairs they win up to 1.5x (4001 rows, us, single / pairs: 28672 x 4096 1.10x,
// 4096 x 14336 1.12x; 512 rows 1.19x both), 18 shapes lose 3 to 11 %; always pairs lost more than 3 % in 1550 (K = 256, 1000 rows: 20 %; 11008 x 4096, 320
// rows: 29 %).
// In one wave of a model's step, where a product follows a short kernel, pairs are quicker than in a loop of products: decode of 256 rows, four layers without
// adapters 1042 -> 1029 us, with a hundred 1715 -> 1662 (in a loop 4096 to 8192 features x 4096 lose 2 to 4 %, 11008 and 13824 win 8 to 11 %).
// With adapters of rank `lora_rank` the first tile of a pair waits for the shrink, and a pair holds twice the tile: K of 2048 and ranks of up to 32, and one wave
// (300 rows of one adapter, a pass 1114 -> 1094 us; 200 rows of eight 1184 -> 1146), or the cheaper plan where most pairs have a tile and a half or a
// feature tile of their own (2000 rows 3830 -> 3750; 1000 rows, whose tiles are less, 2190 -> 2225 with pairs everywhere, of rank 64 2440 -> 2520).
constexpr int kPairWaveTokens = 256, kPairWaveLoraTokens = 512;
constexpr double kPairCostFactor = 1.15, kPairCostMore = 4000.0;
static PairPlan choose_pair(int T, int N, int K, int pairs, long long ws_bytes, double single_cost, int lora_rank) {
  PairPlan plan = pair_plan(T, N, K, pairs, ws_bytes);
  const int tiles_a = (N + 255) / 256, tiles = plan.bn > 0 ? tiles_a * ((T + plan.bn - 1) / plan.bn) : 0;
  const bool cheaper = plan.cost * kPairCostFactor + kPairCostMore < single_cost;
  const bool wave = K >= 2048 && tiles_a >= 16 && tiles <= pairs && ws_bytes > 0 && T <= (lora_rank > 0 ? kPairWaveLoraTokens : kPairWaveTokens);
  bool take = cheaper || wave;
  if (lora_rank > 0) take = lora_rank <= 32 && K >= 2048 && (wave || (cheaper && (tiles_a >= pairs || 2 * tiles >= 3 * pairs)));
  if (!take) plan.bn = 0;
  return plan;
}

}  // namespace lx
