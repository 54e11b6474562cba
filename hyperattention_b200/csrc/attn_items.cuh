// Work items of the tensor-core attention kernels: pairs of query tiles with the list of key tiles they share, and what the loader
// warps do to fetch them.
#pragma once
#include "attn_index.cuh"
#include "tensor_map.cuh"

namespace ha {

struct AttnPlan {
  FastDiv by_pairs, by_segs, by_heads, by_group, by_block;     // pairs, segs_per_head, H, kv_group, window tiles per block
  int n_items, pairs;                 // items = pairs of query tiles x segments
  int tiles, rows;                    // contiguous rows may be loaded as TMA boxes / indexed rows of q (1) and k (2) by gather4
  int row_sb[2], row_sh[2], row_sn[2];   // row maps of q, k: steps of the row number per batch, head and row
};

// One item: query tiles qt0, qt0 + 1 (has1) of segment seg and their common list of key tiles.  Entries [lo_g, hi_g) of the list are
// window (or contiguous) tiles of query tile g; entries n_win .. n_list - 1 are sampled tiles, which both take.  n_list = 0: the end.
struct AttnItem {
  int seg, qt0, has1, n_list;
  int n_win, lo1, hi0, hi1;           // (lo of query tile 0 is 0)
  int first, b, h, hk;                // sorted position of list entry 0 (hyper)
  int q_row0, k_row0, kseg, q_pos0;   // q_pos0: sorted position of query tile qt0's first row (hyper)
  __device__ __forceinline__ int lo(int g) const { return g ? lo1 : 0; }
  __device__ __forceinline__ int hi(int g) const { return g ? hi1 : hi0; }
  __device__ __forceinline__ bool active(int g, int e) const { return (g == 0 || has1) && ((e >= lo(g) && e < hi(g)) || e >= n_win); }
  __device__ __forceinline__ int first_entry(int g) const { return hi(g) > lo(g) ? lo(g) : n_win; }
  __device__ __forceinline__ int last_entry(int g) const { return n_list > n_win ? n_list - 1 : hi(g) - 1; }
  __device__ __forceinline__ int count(int g) const { return (g == 0 || has1) ? hi(g) - lo(g) + n_list - n_win : 0; }
};

// by_keys: enumerate the pairs of smooth windows per KEY tile with the forward's window formula, as the reference's backward does
// (src/hyper_attn_triton.py:290-325): key tile t meets the sorted queries [128 t - 64 (bs - 1), ...); the query tiles are then
// shifted by half a tile when bs is even.  Needs whole blocks (m_k a multiple of bs tiles).
__device__ __forceinline__ AttnItem attn_item(const ha_attn_params& p, const AttnPlan& pl, int item, bool flash, bool by_keys = false) {
  AttnItem it;
  it.seg = pl.by_pairs(item);
  int pr = item - it.seg * pl.pairs;
  const int n_qt = (p.m_q + TILE - 1) / TILE;
  if (flash && (p.flags & HA_FLAG_CAUSAL)) {
    // Items grow with the pair.  Long pairs first; with few pairs the order is turned by the segment, so that a CTA, which
    // takes every 148th item, meets all lengths.  Exact causal attention, turned against not (forward): 64 x 32 heads x 2048 rows 1.79 against
    // 2.35 ms, 8 x 32 x 1024 82 against 113 us, where items outnumber CTAs many times; 32 heads x 2048 66 against 53 us, x 4096 168
    // against 150, x 8192 567 against 473, where they do not; 8 heads x 16384 (64 pairs) 545 against 590.  The line at 32 pairs serves the leaves
    // of causal calls (up to 2048 rows, many segments).
    pr = pl.pairs - 1 - pr;
    if (pl.pairs <= 32) pr += it.seg - pl.by_pairs(pr + it.seg) * pl.pairs;
  }
  it.qt0 = 2 * pr;
  it.q_pos0 = it.qt0 * TILE;
  it.has1 = it.qt0 + 1 < n_qt;
  it.first = 0;
  it.lo1 = 0;
  if (flash) {
    const int n_kt = (p.m_k + TILE - 1) / TILE;
    const bool causal = p.flags & HA_FLAG_CAUSAL;
    it.hi0 = causal ? min(it.qt0 + 1, n_kt) : n_kt;
    it.hi1 = causal ? min(it.qt0 + 2, n_kt) : n_kt;
    it.n_win = it.has1 ? it.hi1 : it.hi0;
    it.n_list = it.n_win;
  } else {
    // block windows (block_window) of both tiles
    const int bs = (p.block_size + TILE - 1) / TILE, tiles = p.m_k / TILE;
    const bool smooth = p.flags & HA_FLAG_SMOOTH;
    const int beta0 = pl.by_block(it.qt0), beta1 = pl.by_block(it.qt0 + 1);
    if (smooth) {
      if (by_keys) {
        // key tiles t = qt0 + h - i, i < bs, of query tile qt0, in ascending order; those of qt0 + 1 are one further on
        const int h = (bs - 1) >> 1;
        it.first = TILE * (it.qt0 + h - bs + 1);
        it.q_pos0 -= (TILE / 2) * ((bs - 1) & 1);
        if (it.q_pos0 < 0) it.q_pos0 += p.m_q;
      } else {
        it.first = TILE * it.qt0 - (TILE / 2) * (bs - 1);
      }
      while (it.first < 0) it.first += p.m_k;
    } else {
      it.first = beta0 * bs * TILE;
    }
    it.hi0 = min(bs, tiles - beta0 * bs);
    it.hi1 = it.n_win = it.hi0;
    if (it.has1) {
      // second window: the same one (both tiles in one block), one tile further on (smooth), or the next block's
      it.lo1 = smooth ? 1 : beta1 > beta0 ? it.hi0 : 0;
      it.hi1 = it.lo1 + min(bs, tiles - beta1 * bs);
      it.n_win = max(it.hi0, it.hi1);
    }
    it.n_list = it.n_win + p.sample_size / TILE;
  }
  const int bh = pl.by_segs(it.seg), part = it.seg - bh * p.segs_per_head;
  const int group = p.kv_group > 1 ? p.kv_group : 1;
  it.b = pl.by_heads(bh);
  it.h = bh - it.b * p.H;
  it.hk = pl.by_group(it.h);
  it.q_row0 = part * p.span + p.q_off;
  it.k_row0 = part * p.span + p.k_off;
  it.kseg = group > 1 ? (it.b * pl.by_group(p.H) + it.hk) * p.segs_per_head + part : it.seg;
  return it;
}

// Rows of list entry e: key row of tile row r inside the segment (-1: none).
__device__ __forceinline__ int item_key_row(const ha_attn_params& p, const AttnItem& it, int e, int r, bool flash) {
  if (flash) {
    const int row = e * TILE + r;
    return row < p.m_k ? row : -1;
  }
  if (e < it.n_win) {
    int pos = it.first + e * TILE + r;
    while (pos >= p.m_k) pos -= p.m_k;
    return p.k_idx[(long long)it.kseg * p.m_k + pos];
  }
  const int s = (e - it.n_win) * TILE + r;
  return p.sample_idx ? p.sample_idx[(long long)it.kseg * p.sample_size + s] : s;
}

__device__ __forceinline__ void red_add_v4(float* addr, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void push_copies(uint32_t bar) {      // an arrival once this thread's cp.async copies so far have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// 128 rows of 64 * slabs elements gathered by ONE warp with cp.async: rows[q] = source row of tile row 32 q + lane (-1: zero fill)
__device__ __forceinline__ void warp_gather_tile(uint32_t smem_base, const uint16_t* __restrict__ base, int64_t row_stride, int slabs, int (&rows)[4], int lane) {
  const int chunk = lane & 7;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int rl = 4 * i + (lane >> 3);
      const int src_row = __shfl_sync(0xffffffffu, rows[0], rl);
      const int row = q * 32 + rl;
      const uint32_t dst = smem_base + row * 128 + ((chunk ^ (row & 7)) << 4);
      const uint16_t* src = base + (int64_t)(src_row < 0 ? 0 : src_row) * row_stride + chunk * 8;
      cp_async16(dst, src, src_row >= 0 ? 16u : 0u);
      if (slabs > 1) cp_async16(dst + TILE * 128, src + 64, src_row >= 0 ? 16u : 0u);
    }
    rows[0] = rows[1]; rows[1] = rows[2]; rows[2] = rows[3];
  }
}

// The part of the plan that depends on the sizes only; false: more items than a launch can count.
inline bool plan_items(AttnPlan& pl, const ha_attn_params& p) {
  pl.pairs = ((p.m_q + TILE - 1) / TILE + 1) / 2;
  const long long items = (long long)p.B * p.H * p.segs_per_head * pl.pairs;
  if (items > 0x7fffffffLL) return false;
  pl.n_items = (int)items;
  pl.by_pairs = FastDiv(pl.pairs > 0 ? pl.pairs : 1);
  pl.by_segs = FastDiv(p.segs_per_head);
  pl.by_heads = FastDiv(p.H > 0 ? p.H : 1);
  pl.by_group = FastDiv(p.kv_group > 1 ? p.kv_group : 1);
  pl.by_block = FastDiv(p.mode == HA_MODE_HYPER ? (p.block_size + TILE - 1) / TILE : 1);
  return true;
}
// May tiles of contiguous rows come as TMA boxes?  A box that runs past the end of a segment brings the next segment's rows, where cp.async
// fills with zeros: hidden weights are 0, but 0 times a row that is not finite is not.  (Past the last row of all, the map
// fills with zeros itself.)
inline bool boxes_end_with_segments(const ha_attn_params& p) { return p.segs_per_head == 1 || (p.m_q % TILE == 0 && p.m_k % TILE == 0); }

// Row maps of q (0) and k (1) for tile::gather4.
inline void plan_row_maps(AttnPlan& pl, const ha_attn_params& p, CUtensorMap (&maps)[2], long long n_q, long long n_k) {
  pl.rows = 0;
  const int Hk = p.kv_group > 1 ? p.H / p.kv_group : p.H;
  for (int x = 0; x < 2 && p.mode == HA_MODE_HYPER; ++x) {
    const int heads = x ? Hk : p.H;
    const int64_t sn = x ? p.k_sn : p.q_sn, sh = x ? p.k_sh : p.q_sh, sb = x ? p.k_sb : p.q_sb;
    int64_t pitch = 1;
    if (!encode_row_map(&maps[x], p.dtype, x ? p.k : p.q, p.d, x ? n_k : n_q, heads, p.B, sn, sh, sb, &pitch)) continue;
    pl.rows |= 1 << x;
    pl.row_sn[x] = (int)(sn / pitch);
    pl.row_sh[x] = heads > 1 ? (int)(sh / pitch) : 0;      // (the encoder has seen that every row number fits)
    pl.row_sb[x] = p.B > 1 ? (int)(sb / pitch) : 0;
  }
}

}  // namespace ha
