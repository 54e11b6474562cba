// Work items of the tensor-core attention kernels: pairs of query tiles with the list of key tiles they share, and what the loader
// warps do to fetch them.
#pragma once
#include "attn_index.cuh"
#include "tensor_map.cuh"

namespace ha {

struct AttnPlan {
  FastDiv by_pairs, by_segs, by_heads, by_group, by_block;     // pairs, segs_per_head, H, kv_group, window tiles per block
  int n_items, pairs;                 // items = pairs of query tiles (or key tiles) x segments
  // exact causal attention (plan_order): items of a round, its segments, the segments after the whole rounds; by_length = 0: no rounds, the
  // segments' own order, a segment's places turned by turn times its number
  FastDiv by_round, by_round_segs, by_rest;
  int by_length, turn, round_segs, whole_items, whole_segs, rest_segs;
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

// Exact causal attention: the items of a segment differ in length (place 0: the longest), and CTA c takes items c, c + grid, ... of one
// order.  That order is by length over a round of segments -- as many as make whole turns of the grid (37 for 4, 8, 12 or 16 places and 148
// CTAs) --, then over the segments that are left; every other turn the CTAs take theirs in the opposite direction
// (item_of_turn).  How much more the longest CTA has than the average (up to 32 places and 295 segments, worked out on the host): with six turns of the
// grid or more 1% in half of the cases, 14% at most; with three to six 6% in half of them, 32% at most; below three turns 10 to 90%, where little can be
// dealt out.  Against the segments' own order (segments x places): 64 x 8 4 for 50%, 128 x 6 6 for 40, 128 x 8 6 for 23, 256 x 8 1 for 10, 128 x
// 16 1 for 17.  Training steps, in turn: 16 heads x 12287 x 64 (128 x 6) 894 -> 856 us, 128 x 1920 x 64 442 -> 425, 2 x 16 heads x 8192 x 128 (128 x 8,
// x 16 in the backward) 1355 -> 1309, 256 x 2047 x 128 1488 -> 1446.
// EXACT: may the launch be exact attention?  Kernels of the hyper pattern, whose items are of one length, are compiled without the order: its few
// instructions in the warp that works the items out cost them 0.5 to 3% (32 x 131072 x 64, step: 3286 -> 3250 us; smooth 32 x 16384 630 -> 609;
// weighted 16 x 32768 590 -> 570; forward of 32 x 131072 1124 -> 1118).
template <bool EXACT>
__host__ __device__ __forceinline__ int item_of_turn(const AttnPlan& pl, int turn, int cta, int grid) {
  return turn * grid + (EXACT && pl.by_length && (turn & 1) ? grid - 1 - cta : cta);
}
__host__ __device__ __forceinline__ int causal_place(const AttnPlan& pl, int item, int& seg) {
  int place;
  if (!pl.by_length) {
    seg = pl.by_pairs(item);
    place = item - seg * pl.pairs;
    if (pl.turn) {
      const int by = seg - pl.by_pairs(seg) * pl.pairs;
      place += pl.turn > 0 ? by : -by;
      place += place < 0 ? pl.pairs : place >= pl.pairs ? -pl.pairs : 0;
    }
  } else if (item < pl.whole_items) {
    const int round = pl.by_round(item);
    item -= round * pl.round_segs * pl.pairs;
    place = pl.by_round_segs(item);
    seg = round * pl.round_segs + item - place * pl.round_segs;
  } else {
    item -= pl.whole_items;
    place = pl.by_rest(item);
    seg = pl.whole_segs + item - place * pl.rest_segs;
  }
  return place;
}

// by_keys: enumerate the pairs of smooth windows per KEY tile with the forward's window formula, as the reference's backward does
// (src/hyper_attn_triton.py:290-325): key tile t meets the sorted queries [128 t - 64 (bs - 1), ...); the query tiles are then
// shifted by half a tile when bs is even.  Needs whole blocks (m_k a multiple of bs tiles).
__device__ __forceinline__ AttnItem attn_item(const ha_attn_params& p, const AttnPlan& pl, int item, bool flash, bool by_keys = false) {
  AttnItem it;
  int pr;
  if (flash && (p.flags & HA_FLAG_CAUSAL)) {
    pr = pl.pairs - 1 - causal_place(pl, item, it.seg);
  } else {
    it.seg = pl.by_pairs(item);
    pr = item - it.seg * pl.pairs;
  }
  const int n_qt = (p.m_q + TILE - 1) / TILE;
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
// The segments' own order: by how much a segment's places are turned against the segment's before.  A CTA takes every 148th item, and should meet all
// lengths on its way.  Unturned, its place advances by 148 mod places a turn, which goes evenly round all of an odd number of places, but only meets
// one in 2 or 4 of an even one.  Turned, the place advances by some fraction more or less, and what decides between up and down is whether a few
// such steps come back to where they began (22 places, up: 22.7 a turn, which is no step at all; 16, down: three steps are one round).  Longest CTA
// over the average, mean of 297 to 1024 segments, down / up / unturned: 5 places 1.15 / 1.18 / 1.07, 7 1.10 / 1.11 / 1.08, 8 1.07 / 1.07 / 1.35, 14
// 1.05 / 1.09 / 1.10, 16 1.10 / 1.05 / 1.20, 19 1.04 / 1.16 / 1.03, 22 1.04 / 1.09 / 1.07.  Forward of 512 x 1152 x 128 239 / 245 / 237 us, of
// 320 x 4864 x 128 1930 / 2228 / 1903, of 320 x 4096 x 128 1577 / 1370 down / up.  Beyond 32 places: unturned.
inline int own_order_turn(int places) {
  if (places > 32 || (places % 2 == 1 && places < 20)) return 0;
  constexpr uint32_t DOWN = 1u << 14 | 1u << 18 | 1u << 22 | 1u << 23 | 1u << 31;
  return places < 32 && (DOWN >> places & 1) ? -1 : 1;
}
// The order of the items (causal_place) for a launch of `grid` CTAs; after n_items and pairs.  width: bytes of an element of the rows that the items of
// a segment share: K and V (2) in the forward, fp32 sums (4) in the backward.  All of a round, and all that is left after the rounds, is live at once,
// and what leaves L2 (126 MB) costs more than the balance gives.  By length against the segments' own order: forward of 64 x 2048 x 128 (67 MB)
// 82 / 111 us, 32 x 4096 x 128 (67) 141 / 204, 32 x 8192 x 128 (134) 507 / 590, 64 x 8192 x 128 (155, one round of 37) 1012 / 1065; backward of 38 x
// 4096 x 128 (159) 546 / 635, 85 x 3072 x 128 (151, after the rounds) 747 / 795, 85 x 6144 x 64 (151, so too) 1394 / 1537, 64 x 8192 x 64 (155) 1785 /
// 1944; 128 x 1920 x 128 (251) 679 / 619, 230 x 1920 x 128 (291) 1244 / 1063.  Odd numbers of places are even enough in the segments' own order to
// want a lower line: forward of 140 x 1664 x 128 (119) 134 / 125, 128 x 1152 x 128 (75) 66 / 70.  With more than two segments a CTA the segments'
// own order is even enough: rounds cost 1 to 3% there (2048 x 2048 x 64, step of 32 heads x 131072:
// 18.97 -> 19.56 ms; 512 x 2048 x 128, forward: 1795 -> 1814 us).
inline void plan_order(AttnPlan& pl, const ha_attn_params& p, int grid, int width) {
  pl.by_length = 0;
  pl.turn = own_order_turn(pl.pairs);
  if (p.mode != HA_MODE_FLASH || !(p.flags & HA_FLAG_CAUSAL) || grid <= 0) return;
  int a = grid, b = pl.pairs;
  while (b) { const int r = a % b; a = b; b = r; }          // a: greatest common divisor
  const int segs = pl.n_items / pl.pairs;
  pl.round_segs = grid / a;
  const long long round_items = (long long)pl.round_segs * pl.pairs, over = (long long)pl.n_items - 2 * grid;      // (two turns at least stay for the rest)
  const int rounds = over > 0 ? (int)(over / round_items) : 0;
  pl.whole_segs = rounds * pl.round_segs;
  pl.whole_items = pl.whole_segs * pl.pairs;
  pl.rest_segs = segs - pl.whole_segs;
  pl.by_round = FastDiv((uint32_t)round_items);
  pl.by_round_segs = FastDiv(pl.round_segs);
  pl.by_rest = FastDiv(pl.rest_segs);
  const long long at_a_time = rounds > 0 && pl.round_segs > pl.rest_segs ? pl.round_segs : pl.rest_segs;
  const long long shared = at_a_time * p.m_k * (p.d + p.dv) * width / (p.kv_group > 1 ? p.kv_group : 1);
  pl.by_length = segs <= 2 * grid && shared <= (long long)(pl.pairs % 2 ? 32 * width : 160) << 20;
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
