// Ragged causal prefill attention over the paged KV cache on the 5th-generation tensor cores.
//
// One CTA = one 64-query tile of one sequence x TWO or FOUR query heads of the same KV group: the 128 rows of a tcgen05 M tile are
// (head, query) pairs of two heads, a CTA has NT = 1 or 2 such tiles (two where the group's heads divide by four and there is more than
// a wave of them), and a K / V block is staged once for all of them.  Keys are walked in blocks of 128 (four cache pages):
//
//   loader  (warp 0, one lane)  Q by TMA from the projection output; K and V pages by TMA straight from the paged cache
//                               through one 5-D tensor map {d, slot, K|V, kv head, block}: the block table supplies the last
//                               coordinate, so pages need not be contiguous; rings of two stages for K and for V
//   MMA     (warp 1)            S = Q K^T into TMEM, O_j = P_j V_j into TMEM; P is a TMEM operand in the columns that its scores had.
//                               Two tiles take turns: P V and the next S of one run while the other's softmax does.  A single tile has
//                               two buffers of S and of O in their place: the next S and P V run while its softmax does
//   softmax (a warpgroup per tile)  one thread per row: scores from TMEM with tcgen05.ld, scale / softcap / ALiBi / causal and
//                               window mask, running max and sum, exp2, P as bf16 back into TMEM; the per-block products O_j come
//                               from TMEM and are folded into fp32 registers with the usual rescaling, so nothing in TMEM ever has
//                               to be rescaled
//
// What bounds it: per tile and block 128 x 128 exponentials take 1024 cycles of the special function units and the products about 1550 of
// the tensor core (S 950: at N = 128 both operands come from shared memory at its full rate; P V 600).  Two tiles fill each other's gaps, and P in
// TMEM spares the stores and half of P V's shared memory.  Launches in a row, 32 heads, one tile per CTA and P through shared memory -> this: 8 KV
// heads, 8192 tokens 1022 -> 597 us, seven prompts of 571 106 -> 62, three of 570 52 -> 32 (two tiles a CTA); 500 tokens 19.8 -> 15.0, 123 10.4 -> 9.5;
// 16 KV heads, 8192 tokens 1046 -> 798, capped 1640 -> 1430, with a bias 3000 -> 2510 (one).  8192 tokens on their own 579, 368 without the softmax.
//
// WIDE: the softmax weights stay fp32 up to the value product: each is split into two bf16 terms, value and remainder, side by side in
// TMEM, and P V is two products into the same accumulator (the layer-by-layer designs ask for it).
//
// Plain, chunked and prefix-cached prefill are one path: `cache_lens` says how many keys precede the chunk.  It replaces the
// flash-attn-2 varlen call of the reference (server/lorax_server/utils/flash_attn.py:180-201) and the mma.sync kernel in
// attention.cu, which stays for head sizes and group sizes this one does not take (d != 128, odd heads per KV head).
// Every wait is bounded and reports through the status word.
#include "attn_tail.cuh"

namespace lx {

constexpr int kFaPage = 32;
constexpr int kFaQ = 64;            // queries per CTA (per head)
constexpr int kFaKeys = 128;        // keys per block
constexpr int kFaD = 128;
constexpr float kFaLog2e = 1.4426950408889634f;

struct FaParams {
  const int* block_tables;
  int max_blocks;
  const int* cu_q;
  const int* cache_lens;
  const int* tile_seq;
  const int* tile_q0;
  __nv_bfloat16* out;
  long long ldo;
  int nh, nkv, group;
  int window;
  float scale, softcap;
  const float* alibi;
  int* status;
  AttnTail tail;
};

template <int NT>
struct FaShape {
  static constexpr int kThreads = 128 * (1 + NT);            // loader, MMA and two idle warps; four softmax warps per tile
  static constexpr int kQBytes = 128 * kFaD * 2;             // of a tile: two 64-wide halves of [128 rows x 64]
  static constexpr int kKBytes = kFaKeys * kFaD * 2;
  static constexpr int kVBytes = kFaKeys * kFaD * 2;
  static constexpr int kTotal = NT * kQBytes + 2 * (kKBytes + kVBytes) + 512 + 1024;
  static constexpr uint32_t kTmemCols = 512;                 // S (later P) of every tile, or of a tile's even and odd blocks, then O alike
  static constexpr int kAhead = 3 - NT;                      // blocks of a tile whose scores may be under way
};

// 5-D tiled load: the paged cache {d, slot in page, K|V, kv head, block}.
LX_DEVICE void tma_load_5d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

LX_DEVICE float fa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
LX_DEVICE float fa_max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// Two fp32 numbers in one 64-bit register: one instruction adds or multiplies both (the same roundings as two).
LX_DEVICE unsigned long long fa_pair(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
LX_DEVICE float2 fa_unpair(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
LX_DEVICE unsigned long long fa_add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
LX_DEVICE unsigned long long fa_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
LX_DEVICE unsigned long long fa_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// The wait for tcgen05.ld as something the loaded registers pass through: their first use stays behind it while other loads are in flight.
LX_DEVICE void fa_wait_ld(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                 "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
LX_DEVICE void fa_wait_ld(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                 "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                 "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]),
                 "+r"(r[31])
               :
               : "memory");
}
template <int N>
LX_DEVICE void fa_regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
LX_DEVICE void fa_regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// How a raw product becomes a score in the log2 domain (the softmax uses exp2): scaled; scaled and capped; also with an ALiBi bias.
enum FaScores : int { kFaPlain = 0, kFaCap = 1, kFaBias = 2 };
struct FaScore {
  float scale_l2, cap_l2, cap_k, slope_l2;       // scale * log2(e), cap * log2(e) (0: none), 2 scale log2(e) / cap, slope * log2(e)
  template <int MODE>
  LX_DEVICE float of(float s, int key) const {
    if (MODE == kFaPlain) return s * scale_l2;
    if (MODE == kFaCap) return softcap_score(s, cap_l2, cap_k);
    return fmaf(slope_l2, (float)key, cap_l2 > 0.f ? softcap_score(s, cap_l2, cap_k) : s * scale_l2);
  }
};

// The keys a row sees, [lo, hi), and what that is over the rows of its warp: chunks of keys that all of them see, or none, need no mask.
struct FaBounds {
  int lo, hi, lo_max, lo_min, hi_min, hi_max;
  LX_DEVICE bool all(int key, int n) const { return key >= lo_max && key + n <= hi_min; }
  LX_DEVICE bool none(int key, int n) const { return key >= hi_max || key + n <= lo_min; }
};

// Products of keys a row does not see become -inf where they lie: their weights are exact zeros without a mask in the passes that follow
// (a block at a tile's edges only, so its code is small rather than quick: a CTA of a short prompt fetches all its code for a block or two).
LX_DEVICE void fa_block_mask(uint32_t ts, int kb0, const FaBounds& bd) {
#pragma unroll 1
  for (int c = 0; c < kFaKeys; c += 16) {
    if (bd.all(kb0 + c, 16)) continue;
    const int lo = bd.lo - (kb0 + c), hi = bd.hi - (kb0 + c);
    uint32_t r[16];
    if (!bd.none(kb0 + c, 16)) {
      tmem_ld_32x32b_x16(ts + (uint32_t)c, r);
      fa_wait_ld(r);
    }
    uint32_t w[8];
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
#pragma unroll
      for (int q = 0; q < 8; ++q) w[q] = (h + q >= lo && h + q < hi) ? r[h + q] : 0xff800000u;
      tmem_st_32x32b_x8(ts + (uint32_t)(c + h), w);
    }
  }
  tc_wait_st();
}

// Maximum over the 128 scores of a row (log2 domain).  Without a bias the scores grow with the products (scale > 0), so the largest product
// gives it.  Plain products have their masked keys at -inf already; MASK: keys outside the bounds do not count.  The code of capped and biased scores
// here and in fa_block_probs is a rolled loop: a CTA of a short prompt fetches all its code for a block or two (unrolled, with and without masks:
// 250 tokens of 32 heads with a bias 19 us -> 27).  Blocks that all rows see whole take capped scores without a mask (with it, 8192 tokens of 16 KV heads
// 1640 us -> 2030); those with a bias, which are formed twice, gain nothing by that.
template <int MODE, bool MASK>
LX_DEVICE float fa_block_max(uint32_t ts, int kb0, const FaBounds& bd, const FaScore& sc) {
  float bm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if constexpr (MODE != kFaBias && !MASK) {
    auto take = [&](const uint32_t (&r)[32]) {
#pragma unroll
      for (int q = 0; q < 32; q += 2) bm[(q >> 1) & 3] = fa_max3(bm[(q >> 1) & 3], __uint_as_float(r[q]), __uint_as_float(r[q + 1]));
    };
    uint32_t ra[32], rb[32];
    tmem_ld_32x32b_x32(ts, ra);
    fa_wait_ld(ra);
    tmem_ld_32x32b_x32(ts + 32u, rb);
    take(ra);
    fa_wait_ld(rb);
    tmem_ld_32x32b_x32(ts + 64u, ra);
    take(rb);
    fa_wait_ld(ra);
    tmem_ld_32x32b_x32(ts + 96u, rb);
    take(ra);
    fa_wait_ld(rb);
    take(rb);
  } else {
#pragma unroll 1
    for (int c = 0; c < kFaKeys; c += 32) {
      if (bd.none(kb0 + c, 32)) continue;
      const int lo = bd.lo - (kb0 + c), hi = bd.hi - (kb0 + c);
      uint32_t r[32];
      tmem_ld_32x32b_x32(ts + (uint32_t)c, r);
      fa_wait_ld(r);
#pragma unroll
      for (int q = 0; q < 32; q += 2) {
        float t[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          t[u] = MODE == kFaBias ? sc.of<MODE>(__uint_as_float(r[q + u]), kb0 + c + q + u) : __uint_as_float(r[q + u]);
          t[u] = (q + u >= lo && q + u < hi) ? t[u] : -INFINITY;
        }
        bm[(q >> 1) & 3] = fa_max3(bm[(q >> 1) & 3], t[0], t[1]);
      }
    }
  }
  const float m = fmaxf(fa_max3(bm[0], bm[1], bm[2]), bm[3]);
  return MODE == kFaBias || m == -INFINITY ? m : sc.of<MODE>(m, 0);
}

// p = exp2(score - m_new) for the 128 keys of the block -> bf16 as a TMEM operand in the columns of the scores: those of 16 keys give
// eight columns of weights (WIDE: and eight of the remainders).  Returns the row sum.  Plain scores: the exponentials of the next 16 keys are
// under way while those before are summed, rounded and stored (one after the other 2360 cycles a block, 1024 of them the special function unit's).
template <int MODE, bool MASK, bool WIDE>
LX_DEVICE float fa_block_probs(uint32_t ts, int kb0, const FaBounds& bd, float m_new, const FaScore& sc) {
  float sum = 0.f;
  const float neg_m = (m_new == -INFINITY) ? 0.f : -m_new;
  auto finish = [&](const float* e, int c) {
    uint32_t pk[8], rest[8];
#pragma unroll
    for (int q = 0; q < 16; q += 2) {
      sum += e[q] + e[q + 1];
      pk[q >> 1] = pack_bf16x2(e[q], e[q + 1]);
      if constexpr (WIDE) {
        const float2 h = unpack_bf16x2(pk[q >> 1]);
        rest[q >> 1] = pack_bf16x2(e[q] - h.x, e[q + 1] - h.y);
      }
    }
    tmem_st_32x32b_x8(ts + (uint32_t)c, pk);
    if constexpr (WIDE) tmem_st_32x32b_x8(ts + (uint32_t)(c + 8), rest);
  };
  if constexpr (MODE == kFaPlain) {
    const unsigned long long scale2 = fa_pair(sc.scale_l2, sc.scale_l2), neg2 = fa_pair(neg_m, neg_m);
    auto exps = [&](const uint32_t (&r)[16], float (&e)[16]) {
#pragma unroll
      for (int q = 0; q < 16; q += 2) {
        const float2 x = fa_unpair(fa_fma2(fa_pair(__uint_as_float(r[q]), __uint_as_float(r[q + 1])), scale2, neg2));
        e[q] = fa_ex2(x.x);
        e[q + 1] = fa_ex2(x.y);
      }
    };
    uint32_t ra[16], rb[16];
    float ea[16], eb[16];
    tmem_ld_32x32b_x16(ts, ra);
    fa_wait_ld(ra);
    tmem_ld_32x32b_x16(ts + 16u, rb);
    exps(ra, ea);
#pragma unroll 1
    for (int c = 0; c < kFaKeys - 32; c += 32) {
      fa_wait_ld(rb);
      tmem_ld_32x32b_x16(ts + (uint32_t)(c + 32), ra);
      exps(rb, eb);
      finish(ea, c);
      fa_wait_ld(ra);
      tmem_ld_32x32b_x16(ts + (uint32_t)(c + 48), rb);
      exps(ra, ea);
      finish(eb, c + 16);
    }
    fa_wait_ld(rb);
    exps(rb, eb);
    finish(ea, kFaKeys - 32);
    finish(eb, kFaKeys - 16);
  } else {
#pragma unroll 1
    for (int c = 0; c < kFaKeys; c += 32) {
      float e[32];
      if (MASK && bd.none(kb0 + c, 32)) {
#pragma unroll
        for (int q = 0; q < 32; ++q) e[q] = 0.f;
      } else {
        const int lo = bd.lo - (kb0 + c), hi = bd.hi - (kb0 + c);
        uint32_t r[32];
        tmem_ld_32x32b_x32(ts + (uint32_t)c, r);
        fa_wait_ld(r);
#pragma unroll
        for (int q = 0; q < 32; ++q) {
          const float x = fa_ex2(sc.of<MODE>(__uint_as_float(r[q]), kb0 + c + q) + neg_m);
          e[q] = !MASK || (q >= lo && q < hi) ? x : 0.f;
        }
      }
      finish(e, c);
      finish(e + 16, c + 16);
    }
  }
  return sum;
}

template <bool WIDE, int NT>
__global__ void __launch_bounds__(FaShape<NT>::kThreads, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv, const FaParams p) {
  using S = FaShape<NT>;
  extern __shared__ uint8_t fa_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(fa_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sq = smem;
  uint8_t* sk = sq + NT * S::kQBytes;
  uint8_t* sv = sk + 2 * S::kKBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sv + 2 * S::kVBytes);
  uint64_t* q_full = bars;            // 1
  uint64_t* k_full = bars + 1;        // 2
  uint64_t* k_empty = bars + 3;       // 2
  uint64_t* v_full = bars + 5;        // 2
  uint64_t* v_empty = bars + 7;       // 2
  uint64_t* s_full = bars + 9;        // per tile; of a single tile, of its even and its odd blocks
  uint64_t* p_full = bars + 11;       // alike, an arrival per softmax warp: weights written, the product before in their columns' O folded
  uint64_t* pv_full = bars + 13;      // alike
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head_groups = p.nh / (2 * NT);
  const int tile = ((int)gridDim.x - 1 - (int)blockIdx.x) / head_groups;      // later tiles of a sequence see more keys: start the long ones first
  const int hc = (int)blockIdx.x % head_groups * 2 * NT;      // first of the CTA's query heads
  const int kvh = hc / p.group;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&pv_full[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_kv);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, S::kTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  const int b = p.tile_seq[tile];
  const int q0 = p.tile_q0[tile];
  const int tok_base = p.cu_q[b];
  const int qlen = p.cu_q[b + 1] - tok_base;
  const int cache = p.cache_lens[b];
  // keys the tile needs: [key_lo, key_hi)
  const int last_q = min(q0 + kFaQ - 1, qlen - 1);
  const int key_hi = cache + last_q + 1;
  const int key_lo = p.window > 0 ? max(cache + q0 + 1 - p.window, 0) : 0;
  const int t_lo = key_lo / kFaKeys;
  const int nblk = max((key_hi + kFaKeys - 1) / kFaKeys - t_lo, 0);
  const int total_pages = (key_hi + kFaPage - 1) / kFaPage;

  if (warp < 4) {
    if constexpr (NT == 2) fa_regs_dec<56>();      // 128 * 56 + 256 * 224 = 384 * 168: what the block was launched with
    if (warp == 0 && lane == 0 && nblk > 0) {
      // Q: rows 0..63 of a tile = its first head, rows 64..127 = its second; two 64-wide halves of d
      mbar_expect_tx(q_full, (uint32_t)(NT * S::kQBytes));
      for (int g = 0; g < 2 * NT; ++g)
        for (int hf = 0; hf < 2; ++hf)
          tma_load_2d(sq + (g >> 1) * S::kQBytes + hf * 16384 + (g & 1) * 8192, &tmap_q, q_full, (hc + g) * kFaD + hf * 64, tok_base + q0);
      const int* bt = p.block_tables + (long long)b * p.max_blocks;
      for (int j = 0; j < nblk; ++j) {
        const int st = j & 1;
        int blk[4];
        for (int pg = 0; pg < 4; ++pg) {
          const int page = (t_lo + j) * 4 + pg;
          blk[pg] = (page < total_pages && page < p.max_blocks) ? bt[page] : 0;      // a page past the keys reads block 0: masked, but finite
        }
        for (int kv = 0; kv < 2; ++kv) {
          uint64_t* full = kv ? &v_full[st] : &k_full[st];
          if (!mbar_wait(kv ? &v_empty[st] : &k_empty[st], ((j >> 1) & 1) ^ 1, abort_flag)) {
            report_status(p.status, kTimeoutEmptyBarrier, tile);
            *abort_flag = 1;
            j = nblk;
            break;
          }
          uint8_t* dst = kv ? sv + st * S::kVBytes : sk + st * S::kKBytes;
          mbar_expect_tx(full, (uint32_t)S::kKBytes);
          for (int pg = 0; pg < 4; ++pg)
            for (int hf = 0; hf < 2; ++hf) tma_load_5d(dst + hf * 16384 + pg * 4096, &tmap_kv, full, hf * 64, 0, kv, kvh, blk[pg]);
        }
      }
    } else if (warp == 1 && nblk > 0) {
      // The whole warp walks the blocks and one lane issues: addresses and descriptors stay uniform, so that MMAs of 64 cycles each
      // are not held up by their issue (all of it by one lane of a divergent warp: 8192 tokens 615 us instead of 579).
      const uint32_t idesc_s = make_idesc(128, kFaKeys, kFmtBF16, kFmtBF16);
      const uint32_t idesc_pv = make_idesc(128, kFaD, kFmtBF16, kFmtBF16, 0, 1);          // B (= V) is MN-major
      const uint64_t dq = make_desc_k_sw128(smem_u32(sq)), dk = make_desc_k_sw128(smem_u32(sk)), dv = make_desc_mn_sw128(smem_u32(sv), 16384, 1024);
      const bool leader = elect_one();
      auto give_up = [&](int code) {
        if (leader) report_status(p.status, code, tile);
        *abort_flag = 1;
      };
      // S of tile t and block j.  It takes the columns of the weights that a product issued before it reads: one thread's MMAs run in order.
      auto issue_s = [&](int t, int j) {
        const int at_s = NT == 2 ? t : j & 1;
        const uint64_t da = dq + (uint64_t)((t * S::kQBytes) >> 4), db = dk + (uint64_t)(((j & 1) * S::kKBytes) >> 4);
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < kFaD / 16; ++ks) {
            const uint64_t at = (uint64_t)((ks >> 2) * (16384 >> 4) + (ks & 3) * 2);
            umma_f16_ss(tmem_base + (uint32_t)(at_s * 128), da + at, db + at, idesc_s, ks > 0 ? 1u : 0u);
          }
          tc_commit(&s_full[at_s]);
          if (t == NT - 1) tc_commit(&k_empty[j & 1]);
        }
        __syncwarp();
      };
      bool ok = mbar_wait(q_full, 0, abort_flag) && mbar_wait(&k_full[0], 0, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) give_up(kTimeoutFullBarrier);
      tc_fence_after();
#pragma unroll
      for (int t = 0; t < NT; ++t)
        if (ok) issue_s(t, 0);
      if (NT == 1 && ok && nblk > 1) {
        ok = __all_sync(0xffffffffu, mbar_wait(&k_full[1], 0, abort_flag));
        if (!ok) give_up(kTimeoutFullBarrier);
        tc_fence_after();
        if (ok) issue_s(0, 1);
      }
      for (int j = 0; ok && j < nblk; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(&v_full[j & 1], (j >> 1) & 1, abort_flag));
        if (!ok) { give_up(kTimeoutFullBarrier); break; }
        const uint64_t dvj = dv + (uint64_t)(((j & 1) * S::kVBytes) >> 4);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int at_s = NT == 2 ? t : j & 1;
          ok = __all_sync(0xffffffffu, mbar_wait(&p_full[at_s], NT == 2 ? j & 1 : (j >> 1) & 1, abort_flag));
          if (!ok) { give_up(kTimeoutTmemEmpty); break; }
          tc_fence_after();
          const uint32_t tmem_p = tmem_base + (uint32_t)(at_s * 128), tmem_o = tmem_base + (uint32_t)(256 + at_s * 128);
          if (leader) {
#pragma unroll
            for (int ks = 0; ks < kFaKeys / 16; ++ks) {
              const uint64_t db = dvj + (uint64_t)(ks * (2048 >> 4));
              umma_f16_ts(tmem_o, tmem_p + (uint32_t)(ks * 16), db, idesc_pv, ks > 0 ? 1u : 0u);
              if constexpr (WIDE) umma_f16_ts(tmem_o, tmem_p + (uint32_t)(ks * 16 + 8), db, idesc_pv, 1u);
            }
            tc_commit(&pv_full[at_s]);
            if (t == NT - 1) tc_commit(&v_empty[j & 1]);
          }
          __syncwarp();
          const int next = j + S::kAhead;
          if (next < nblk) {
            if (t == 0) {
              ok = __all_sync(0xffffffffu, mbar_wait(&k_full[next & 1], (next >> 1) & 1, abort_flag));
              if (!ok) { give_up(kTimeoutFullBarrier); break; }
              tc_fence_after();
            }
            issue_s(t, next);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax warps: one row per thread
    if constexpr (NT == 2) fa_regs_inc<224>();
    const int t = (warp >> 2) - 1;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const int head = hc + 2 * t + (row >> 6);
    const int qi = q0 + (row & 63);
    const bool row_ok = qi < qlen;
    const int hi = cache + min(qi, qlen - 1) + 1;      // (a row past the sequence's end sees what its last one does, and is not stored)
    const int lo = (p.window > 0 && hi > p.window) ? hi - p.window : 0;
    const FaBounds bd{lo, hi, __reduce_max_sync(0xffffffffu, lo), __reduce_min_sync(0xffffffffu, lo), __reduce_min_sync(0xffffffffu, hi),
                      __reduce_max_sync(0xffffffffu, hi)};
    FaScore sc;
    sc.scale_l2 = p.scale * kFaLog2e;
    sc.cap_l2 = p.softcap > 0.f ? p.softcap * kFaLog2e : 0.f;
    sc.cap_k = p.softcap > 0.f ? 2.f * sc.scale_l2 / p.softcap : 0.f;
    sc.slope_l2 = p.alibi != nullptr ? p.alibi[head] * kFaLog2e : 0.f;
    // (the plain forms take the largest product for the largest score)
    const int mode = p.alibi != nullptr || !(p.scale > 0.f) ? kFaBias : p.softcap > 0.f ? kFaCap : kFaPlain;
    const uint32_t trow = tmem_base + ((uint32_t)(quad * 32) << 16);
    // where block j's scores and product lie, and which of the tile's barriers (and what parity) say that they are complete
    auto part = [&](int j) { return NT == 2 ? t : j & 1; };
    auto parity = [&](int j) { return (uint32_t)(NT == 2 ? j & 1 : (j >> 1) & 1); };

    float m = -INFINITY, l = 0.f;
    unsigned long long o[kFaD / 2];           // pairs of columns
#pragma unroll
    for (int i = 0; i < kFaD / 2; ++i) o[i] = 0ull;
    // o += the product of block j, relative to the largest score up to it
    auto fold = [&](int j) {
      if (!mbar_wait(&pv_full[part(j)], parity(j), abort_flag)) return false;
      tc_fence_after();
      const uint32_t to = trow + (uint32_t)(256 + part(j) * 128);
      auto add = [&](const uint32_t (&r)[32], int c) {
#pragma unroll
        for (int q = 0; q < 32; q += 2) o[(c + q) >> 1] = fa_add2(o[(c + q) >> 1], fa_pair(__uint_as_float(r[q]), __uint_as_float(r[q + 1])));
      };
      uint32_t ra[32], rb[32];
      tmem_ld_32x32b_x32(to, ra);
      fa_wait_ld(ra);
      tmem_ld_32x32b_x32(to + 32u, rb);
      add(ra, 0);
      fa_wait_ld(rb);
      tmem_ld_32x32b_x32(to + 64u, ra);
      add(rb, 32);
      fa_wait_ld(ra);
      tmem_ld_32x32b_x32(to + 96u, rb);
      add(ra, 64);
      fa_wait_ld(rb);
      add(rb, 96);
      return true;
    };
    bool alive = nblk > 0;
    auto give_up = [&]() {
      report_status(p.status, kTimeoutTmemFull, tile);
      *abort_flag = 1;
      alive = false;
    };

    for (int j = 0; j < nblk && alive; ++j) {
      const int kb0 = (t_lo + j) * kFaKeys;
      // (two tiles: the product of the block before has to leave its columns first, and the other tile's runs meanwhile)
      if (NT == 2 && j > 0 && !fold(j - 1)) { give_up(); break; }
      if (!mbar_wait(&s_full[part(j)], parity(j), abort_flag)) { give_up(); break; }
      tc_fence_after();
      const uint32_t ts = trow + (uint32_t)(part(j) * 128);
      // pass 1: block maximum of this row (log2 domain).  Plain scores have their masked keys set to -inf first, the others are masked chunk
      // by chunk: a capped -inf is finite
      const bool inside = bd.all(kb0, kFaKeys);
      if (mode == kFaPlain && !inside) fa_block_mask(ts, kb0, bd);
      float bm;
      if (mode == kFaPlain) bm = fa_block_max<kFaPlain, false>(ts, kb0, bd, sc);
      else if (mode == kFaCap) bm = inside ? fa_block_max<kFaCap, false>(ts, kb0, bd, sc) : fa_block_max<kFaCap, true>(ts, kb0, bd, sc);
      else bm = fa_block_max<kFaBias, true>(ts, kb0, bd, sc);
      const float m_new = fmaxf(m, bm);
      const float alpha = (m_new == -INFINITY) ? 1.f : fa_ex2(m - m_new);
      // pass 2: weights -> bf16 operand, row sum
      float sum;
      if (mode == kFaPlain) sum = fa_block_probs<kFaPlain, false, WIDE>(ts, kb0, bd, m_new, sc);
      else if (mode == kFaCap) sum = inside ? fa_block_probs<kFaCap, false, WIDE>(ts, kb0, bd, m_new, sc) : fa_block_probs<kFaCap, true, WIDE>(ts, kb0, bd, m_new, sc);
      else sum = fa_block_probs<kFaBias, true, WIDE>(ts, kb0, bd, m_new, sc);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[part(j)]);
      if (NT == 1 && j > 0 && !fold(j - 1)) { give_up(); break; }
      l = l * alpha + sum;
      if (j > 0 && !__all_sync(0xffffffffu, alpha == 1.f)) {      // some row of the warp saw a new maximum
        const unsigned long long alpha2 = fa_pair(alpha, alpha);
#pragma unroll
        for (int i = 0; i < kFaD / 2; ++i) o[i] = fa_mul2(o[i], alpha2);
      }
      m = m_new;
    }
    if (alive) {
      if (mbar_wait(&pv_full[part(nblk - 1)], parity(nblk - 1), abort_flag)) {
        tc_fence_after();
        const uint32_t to = trow + (uint32_t)(256 + part(nblk - 1) * 128);
        const float inv = l > 0.f ? attn_denominator(p.tail, head, m, l) * p.tail.scale : 0.f;
        const __nv_bfloat16* grow = p.tail.gate != nullptr ? p.tail.gate + (long long)(tok_base + qi) * p.tail.ldg + (long long)head * kFaD : nullptr;
        __nv_bfloat16* orow = p.out + (long long)(tok_base + qi) * p.ldo + (long long)head * kFaD;
#pragma unroll
        for (int c = 0; c < kFaD; c += 16) {
          uint32_t r[16];
          tmem_ld_32x32b_x16(to + (uint32_t)c, r);
          fa_wait_ld(r);
          if (row_ok) {
#pragma unroll
            for (int q = 0; q < 16; q += 8) {
              uint32_t w[4];
              float v[8];
#pragma unroll
              for (int u = 0; u < 8; u += 2) {
                const float2 s = fa_unpair(o[(c + q + u) >> 1]);
                v[u] = (s.x + __uint_as_float(r[q + u])) * inv;
                v[u + 1] = (s.y + __uint_as_float(r[q + u + 1])) * inv;
              }
              if (p.tail.turn != nullptr) attn_turn_back8(p.tail, v, c + q, cache + qi);
              if (grow != nullptr) {
                const uint4 g = *reinterpret_cast<const uint4*>(grow + c + q);
                const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const float2 z = unpack_bf16x2(gw[u]);
                  v[2 * u] = __fdividef(v[2 * u], 1.f + __expf(-z.x));
                  v[2 * u + 1] = __fdividef(v[2 * u + 1], 1.f + __expf(-z.y));
                }
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) w[u] = pack_bf16x2(v[2 * u], v[2 * u + 1]);
              *reinterpret_cast<uint4*>(orow + c + q) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      } else {
        report_status(p.status, kTimeoutTmemFull, tile);
        *abort_flag = 1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, S::kTmemCols); }
}

typedef CUresult (*FaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static FaEncodeFn fa_encode_fn() {
  static FaEncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<FaEncodeFn>(ptr);
  }
  return fn;
}

template <bool WIDE, int NT>
static int launch_fa_t(const CUtensorMap& tq, const CUtensorMap& tkv, const FaParams& p, int num_tiles, cudaStream_t s) {
  using S = FaShape<NT>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_tc_kernel<WIDE, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (e != cudaSuccess) return -(int)e;
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  // the heads of a query tile run side by side (they share its keys' pages where they share a KV head), long tiles first
  launch_pdl(attn_prefill_tc_kernel<WIDE, NT>, dim3(num_tiles * (p.nh / (2 * NT))), dim3(S::kThreads), (size_t)S::kTotal, s, tq, tkv, p);
  return -(int)cudaGetLastError();
}
// Two tiles a CTA where the group allows it and single ones would take more than one wave.  In one wave a tile on its own is quicker, in two it is not:
// 32 heads, us, one / two tiles a CTA: 123 tokens 9.5 / 12.3, 500 (128 CTAs of one) 15.0 / 18.8, capped 20.5 / 28.4; three prompts of 300 (240) 20.5 /
// 16.4, capped 25.0 / 22.2; five of 100 behind 500 keys (160) 30.4 / 22.7.  One prompt of 640 to 1000 (160 to 256), whose CTAs are of unequal length, 17.6 / 21.1 to
// 28.1 / 29.3.
constexpr long long kFaSpreadTiles = 148;
template <bool WIDE>
static int launch_fa(const CUtensorMap& tq, const CUtensorMap& tkv, const FaParams& p, int num_tiles, cudaStream_t s) {
  return p.group % 4 == 0 && (long long)num_tiles * (p.nh / 2) > kFaSpreadTiles ? launch_fa_t<WIDE, 2>(tq, tkv, p, num_tiles, s)
                                                                               : launch_fa_t<WIDE, 1>(tq, tkv, p, num_tiles, s);
}

static int attn_prefill_tc(const void* q, long long ldq, int T, const void* kv, int num_blocks, const int* block_tables, int max_blocks,
                           const int* cu_q, const int* cache_lens, const int* tile_seq, const int* tile_q0, int num_tiles, void* out,
                           long long ldo, int nh, int nkv, int window, float scale, float softcap, const float* alibi, int wide,
                           const AttnTail& tail, int* status, void* stream) {
  if (num_tiles <= 0) return 0;
  FaEncodeFn fn = fa_encode_fn();
  if (fn == nullptr) return -2;
  CUtensorMap tq, tkv;
  {
    cuuint64_t dims[2] = {(cuuint64_t)nh * kFaD, (cuuint64_t)T};
    cuuint64_t strides[1] = {(cuuint64_t)ldq * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)kFaQ};
    cuuint32_t es[2] = {1, 1};
    if (fn(&tq, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(q), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -3;
  }
  {
    cuuint64_t dims[5] = {(cuuint64_t)kFaD, (cuuint64_t)kFaPage, 2, (cuuint64_t)nkv, (cuuint64_t)num_blocks};
    cuuint64_t strides[4] = {(cuuint64_t)kFaD * 2, (cuuint64_t)kFaPage * kFaD * 2, (cuuint64_t)2 * kFaPage * kFaD * 2,
                             (cuuint64_t)nkv * 2 * kFaPage * kFaD * 2};
    cuuint32_t box[5] = {64, (cuuint32_t)kFaPage, 1, 1, 1};
    cuuint32_t es[5] = {1, 1, 1, 1, 1};
    if (fn(&tkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(kv), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return -4;
  }
  FaParams p{};
  p.block_tables = block_tables; p.max_blocks = max_blocks; p.cu_q = cu_q; p.cache_lens = cache_lens;
  p.tile_seq = tile_seq; p.tile_q0 = tile_q0;
  p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.nh = nh; p.nkv = nkv; p.group = nh / nkv; p.window = window; p.scale = scale; p.softcap = softcap; p.alibi = alibi; p.status = status; p.tail = tail;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return wide ? launch_fa<true>(tq, tkv, p, num_tiles, st) : launch_fa<false>(tq, tkv, p, num_tiles, st);
}

}  // namespace lx

extern "C" {

// 1: the tensor-core kernel takes this shape (d = 128, an even number of query heads per KV head, 16-byte aligned strides).
int lx_attn_prefill_tc_supported(int nh, int nkv, int d, long long ldq, long long ldo) {
  return (d == 128 && nkv > 0 && nh % nkv == 0 && ((nh / nkv) % 2) == 0 && ldq % 8 == 0 && ldo % 8 == 0) ? 1 : 0;
}

// Same contract as lx_attn_prefill_alibi (64-query tiles listed by tile_seq / tile_q0), plus the number of tokens `T` of the q
// buffer and the number of blocks of the cache (bounds of the two tensor maps) and the status word.  wide: fp32 softmax weights.
int lx_attn_prefill_tc(const void* q, long long ldq, int T, const void* kv, int num_blocks, const int* block_tables, int max_blocks,
                       const int* cu_q, const int* cache_lens, const int* tile_seq, const int* tile_q0, int num_tiles, void* out, long long ldo,
                       int nh, int nkv, int d, int window, float scale, float softcap, const float* alibi, int wide, int* status, void* stream) {
  if (!lx_attn_prefill_tc_supported(nh, nkv, d, ldq, ldo)) return -1;
  return lx::attn_prefill_tc(q, ldq, T, kv, num_blocks, block_tables, max_blocks, cu_q, cache_lens, tile_seq, tile_q0, num_tiles, out, ldo, nh, nkv,
                             window, scale, softcap, alibi, wide, lx::AttnTail{}, status, stream);
}

// The same with fp32 softmax weights, a sink per head, outputs turned back, a gate [T, ldg] and a factor on them (gqa.cu has the details).
int lx_gqa_prefill_tc(const void* q, long long ldq, int T, const void* kv, int num_blocks, const int* block_tables, int max_blocks,
                      const int* cu_q, const int* cache_lens, const int* tile_seq, const int* tile_q0, int num_tiles, void* out, long long ldo,
                      int nh, int nkv, int d, int window, float scale, float softcap, const float* sink, const void* gate, long long ldg,
                      float out_scale, const float* turn, int turn_dims, int turn_rows, int* status, void* stream) {
  if (!lx_attn_prefill_tc_supported(nh, nkv, d, ldq, ldo) || turn_dims % 2 != 0 || turn_dims > d || (gate != nullptr && ldg % 8 != 0)) return -1;
  return lx::attn_prefill_tc(q, ldq, T, kv, num_blocks, block_tables, max_blocks, cu_q, cache_lens, tile_seq, tile_q0, num_tiles, out, ldo, nh, nkv,
                             window, scale, softcap, nullptr, 1,
                             lx::AttnTail{sink, reinterpret_cast<const __nv_bfloat16*>(gate), ldg, out_scale, turn, turn_dims, turn_rows}, status, stream);
}

}  // extern "C"
