// The LoRA delta of a short step added where a product's result is formed: y[t, n] += sum_j v[t, part(n) r + j] B_cat[n, j] with B_cat of the row's
// adapter, from the shrink's fp32 v.
#pragma once

#include "common.cuh"

extern "C" {
// What the launch that adds the delta needs: the step's table of (slot, first row, rows <= 32, -), where the slots' B_cat of the projection lie
// (arena + slot_base + rank * unit_off), the shrink's result, and the parts' boundaries along N (multiples of 128).
struct LxLoraAdd {
  const void* tiles;
  int num_tiles, num_slots;
  const void* arena;
  const long long* slot_base;
  const int* slot_rank;
  long long unit_off;
  const float* v;
  int ldv, n0, n1;
  int tables_const;          // no kernel that may still run writes tiles, slot_base, slot_rank and arena: they are read before the wait
  int* status;
};
}

namespace lx {

// v is read 16 bytes at a time (part * rank is a multiple of 16 columns).
inline bool lora_add_aligned(const LxLoraAdd& a) { return a.ldv % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15) == 0; }

constexpr int kLoraAddRows = 256;
struct LoraAddRow {
  const __nv_bfloat16* b;    // B_cat of the row's adapter
  int r;                     // its rank, 0: the base model's row
  int pad_;
};

struct LoraAddEntry { int slot, row0, nrows, pad_; };
LX_DEVICE LoraAddRow lora_add_row_of(const LxLoraAdd& a, int slot) {
  if (slot < 0) return LoraAddRow{nullptr, 0, 0};
  if (slot >= a.num_slots) { report_status(a.status, kBadIndex, slot); return LoraAddRow{nullptr, 0, 0}; }
  const int r = a.slot_rank[slot];
  const long long base = a.slot_base[slot];
  if (r <= 0 || base < 0) return LoraAddRow{nullptr, 0, 0};
  return LoraAddRow{reinterpret_cast<const __nv_bfloat16*>(a.arena) + base + (long long)r * a.unit_off, r, 0};
}

// rows[t] of the step's T <= kLoraAddRows rows, by the whole block.  (A table may be older than the batch: rows past T are gone.)
LX_DEVICE void lora_add_rows(const LxLoraAdd& a, int T, LoraAddRow* rows) {
  for (int t = threadIdx.x; t < T; t += blockDim.x) rows[t] = LoraAddRow{nullptr, 0, 0};
  __syncthreads();
  for (int e = threadIdx.x; e < a.num_tiles; e += blockDim.x) {
    const LoraAddEntry q = reinterpret_cast<const LoraAddEntry*>(a.tiles)[e];
    if (q.slot < 0) continue;
    const LoraAddRow row = lora_add_row_of(a, q.slot);
    for (int t = max(q.row0, 0); t < min(q.row0 + q.nrows, T); ++t) rows[t] = row;
  }
  __syncthreads();
}

// The same for one row t < 32 per lane, by a warp on its own: live entries come first, sorted by row, and hold a row each at least, so the
// first 32 have these rows.
LX_DEVICE LoraAddRow lora_add_row32(const LxLoraAdd& a, int t) {
  const int lane = threadIdx.x & 31;
  LoraAddEntry q{-1, 0, 0, 0};
  if (lane < a.num_tiles) q = reinterpret_cast<const LoraAddEntry*>(a.tiles)[lane];
  int slot = -1;
#pragma unroll 1
  for (int e = 0; e < min(a.num_tiles, 32); ++e) {
    const int es = __shfl_sync(0xffffffffu, q.slot, e), r0 = __shfl_sync(0xffffffffu, q.row0, e), n = __shfl_sync(0xffffffffu, q.nrows, e);
    if (es < 0) break;
    if (t >= r0 && t < r0 + n) slot = es;
  }
  return lora_add_row_of(a, slot);
}
LX_DEVICE int lora_add_part(const LxLoraAdd& a, int n) { return n < a.n0 ? 0 : (n < a.n1 ? 1 : 2); }
// sum + the dot product of eight ranks, in rank order
LX_DEVICE float lora_dot8(uint4 b, float4 v0, float4 v1, float sum) {
  const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y), b2 = unpack_bf16x2(b.z), b3 = unpack_bf16x2(b.w);
  sum = fmaf(v0.x, b0.x, sum); sum = fmaf(v0.y, b0.y, sum);
  sum = fmaf(v0.z, b1.x, sum); sum = fmaf(v0.w, b1.y, sum);
  sum = fmaf(v1.x, b2.x, sum); sum = fmaf(v1.y, b2.y, sum);
  sum = fmaf(v1.z, b3.x, sum); sum = fmaf(v1.w, b3.y, sum);
  return sum;
}

}  // namespace lx
