// Attention forward on 5th-generation tensor cores (tcgen05 + TMEM), bf16 / fp16, head dims 64 and 128: one persistent,
// warp-specialised kernel for both patterns (sorted block windows + sampled rows; exact attention with or without mask).
//
// One CTA of 640 threads per SM walks work items; an item is a PAIR of 128-row query tiles of one segment and the list of
// key tiles the two pair with (AttnItem): every key tile is fetched once for both.  Roles:
//   * softmax groups 0 / 1 (128 threads each; thread = query row = TMEM lane) of the pair's two query tiles: maximum of the row's 64
//     scores of a unit, then P = exp2(S - running maximum) back to TMEM in the input dtype and the row's sum.  The accumulator lives in
//     TMEM; the group whose maximum grew rescales it row by row once its P is stored (the product before has had that long to
//     complete).  The reference is the exact maximum on purpose: the largest weight of a row is then 1, which a 16-bit P holds
//     without rounding.  A reference that lags (up to 2^8) saves most of the rescaling -- 32 x 131072 forward 1.06 instead
//     of 1.14 ms, 16 x 16384 causal 0.58 instead of 0.61 -- but its outputs are 2 to 6% further from 64 bits (32 x 4096: 2.30e-3 instead of
//     2.17e-3).
//   * epilogue group (128 threads): O of a finished query tile -> registers -> normalised, merged with the rows already stored
//     if the call asks for it, stored.  The softmax groups are meanwhile in the next item.
//   * four MMA warps, S = Q K^T and O += P V of either group, one elected lane issuing from warp-uniform code (descriptors in
//     uniform registers: an N = 128 step is accepted every 64 cycles, the tensor pipe's own rate; the same instructions from
//     a divergent lane cost 126).
//   * four loader warps: contiguous rows by TMA boxes, rows named by an index by tile::gather4 (K) or cp.async (V, Q) -- the two
//     paths run side by side (gather4: about 2200 cycles per tile of 128 rows of 128 bytes; one warp's cp.async: about 3000).
//     One of them works out the items and hands their descriptors to everybody through a small ring: the index arithmetic is
//     done once per item and exists once in the code.
// The roles' loops are kept small (rolled over column chunks and groups) because their code shares the SM's instruction caches:
// the same kernel with everything unrolled spent more warp time waiting for instructions than executing them.
// A unit of the chain S -> softmax -> P V is half a key tile (64 keys).  TMEM (512 columns): group g has score buffers of 64
// columns from 256 g on, three (DV = 64) or two (DV = 128), and O behind them; P takes the place of its scores.  S of the
// next units is there before a group asks for it, so a group goes from one unit to the next without waiting.
// What bounds it: the exponential unit (16 a clock and SM: 1024 cycles per 128 x 128 tile), which is why a part of the exponentials
// is computed on the FMA pipe (poly_exp2_2), and at head dim 128 the tensor pipe.
#include "attn_items.cuh"

#include <type_traits>

namespace ha {

template <int D, int DV> struct FwdCfg {
  static constexpr int NB = DV == 64 ? 3 : 2;                    // score buffers (64 keys each) per group
  static constexpr int W = D > DV ? D : DV;
  static constexpr int Q_TILE = TILE * D * 2, KV_TILE = TILE * W * 2;
  static constexpr int NQ = D == 64 ? 4 : 3;                     // query-tile slots
  static constexpr int NKV = W == 64 ? 8 : 4;                    // key/value slots: K tiles in the even, V tiles in the odd ones
  static constexpr int OFF_Q = 0, OFF_KV = NQ * Q_TILE;
  static constexpr int OFF_STAT = OFF_KV + NKV * KV_TILE;        // [group][row]: (reference, sum) of a finished row
  static constexpr int SMEM_USED = OFF_STAT + 2 * TILE * 8;      // from the first 1 KB boundary after the static variables
  static constexpr int COL_O = NB * 64;                          // group g: score buffers at 256 g + 64 b, O behind them
};

namespace fw {
constexpr int THREADS = 640;
constexpr int W_EPI = 8, W_S = 12, W_PV = 14, W_Q = 16, W_K = 17;   // first warp of each role (S, P V, V: two each)
constexpr int ND = 4;                 // descriptor ring
constexpr int CONSUMERS = 19;         // warps that read every descriptor (all but the one that writes it)
enum { B_KV_FULL = 0, B_KV_EMPTY = 8, B_Q_FULL = 16, B_Q_EMPTY = 20, B_S_READY = 24, B_PV_DONE = 30, B_O_FULL = 36, B_P_READY = 38, B_O_FREE = 44,
       B_STAT = 46, B_D_FULL = 48, B_D_EMPTY = 48 + ND, N_BARS = 48 + 2 * ND };      // (S ready, P ready, product done: 3 g + buffer)
}  // namespace fw

struct FwdMaps { CUtensorMap tile[3], rows[2]; };    // tiles of q, k, v; rows of q, k

// KIND: the plain hyper pattern, exact attention, or any call (merging calls, weighted sampling): the code of an instance is what the
// instruction caches have to hold, so the two frequent kinds carry nothing they do not use.
enum { FWD_HYPER = 0, FWD_FLASH = 1, FWD_ANY = 2 };
template <typename T, int D, int DV, int KIND>
__global__ void __launch_bounds__(fw::THREADS, 1) attn_tc_fwd_kernel(const ha_attn_params p, const AttnPlan pl, const __grid_constant__ FwdMaps maps) {
  chain_begin();
  using namespace fw;
  using Cfg = FwdCfg<D, DV>;
  constexpr int NQ = Cfg::NQ, NKV = Cfg::NKV, NB = Cfg::NB;
  const bool flash = KIND == FWD_FLASH || (KIND == FWD_ANY && p.mode == HA_MODE_FLASH);
  constexpr bool WT = KIND == FWD_ANY;                 // weighted sampling / merging possible
  // Pairs of every eight whose exponentials go to the FMA pipe.  It pays where the chain is bound by the exponential unit, i.e. in exact
  // attention (64 x 32 heads x 2048 rows, head dim 64: 1.85 -> 1.79 ms; 32 x 4096: 178 -> 168 us; head dim 128, 8 x 32768: 2.09 -> 2.05 ms); the
  // hyper pattern is bound by its gathers and its rescaling before that (call at 32 x 131072: 1.151 ms without, 1.156 with).
  constexpr int POLY = KIND == FWD_FLASH ? 2 : 0;
  const bool merge = KIND == FWD_ANY && (p.flags & HA_FLAG_MERGE);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t s_base = smem_u32(smem);
  __shared__ __align__(16) AttnItem s_item[ND];
  __shared__ uint64_t bars[N_BARS];
  __shared__ uint32_t tmem_slot;
  __shared__ uint32_t s_issued[4];        // ring positions the loaders have got to
  __shared__ int s_abort;
  __shared__ int s_bail;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (cta_sees_failure(p.status, &s_bail)) return;   // an earlier CTA gave up: drain quickly (uniform over the CTA)
  {
    // should the window start somewhere else than assumed, do nothing rather than run over its end
    uint32_t dyn;
    asm volatile("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    if ((uint32_t)(smem - smem_raw) + (uint32_t)Cfg::SMEM_USED > dyn) {      // uniform over the grid
      if (tid == 0) report_status(p.status, p.status_host, HA_DEV_BAD_LAUNCH);
      return;
    }
  }
  float2* s_stat = reinterpret_cast<float2*>(smem + Cfg::OFF_STAT);
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) -> uint32_t { return bar0 + 8 * i; };
  if (tid == 0) {
    // arrivals per phase: 32 (every lane of the tile's loader) on the tiles' "full" barriers, 128 (a group) on the hand-offs of the
    // thread groups, one per reading warp on "descriptor empty", 2 (both groups' MMA warps) on the tiles' "empty" barriers, 1 (a
    // tcgen05.commit, the scheduler) elsewhere
    for (int i = 0; i < N_BARS; ++i) {
      const bool loader = (i >= B_KV_FULL && i < B_KV_EMPTY) || (i >= B_Q_FULL && i < B_Q_EMPTY);
      const bool group = i >= B_P_READY && i < B_D_FULL;
      mbar_init(bar(i), loader ? 32 : group ? 128 : i >= B_D_EMPTY ? CONSUMERS : i >= B_KV_EMPTY && i < B_Q_FULL ? 2 : 1);
    }
    s_abort = 0;
    mbar_fence_init();
  }
  if (warp == W_S) tmem_alloc(smem_u32(&tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // A wait that gives up (or finds the abort flag up) ends the role's loop; the status word is set once, at the end.  Called by whole
  // warps; one answer for the warp.
  auto wait = [&](int b, uint32_t parity) -> bool { return __all_sync(0xffffffffu, mbar_wait_or_abort(bar(b), parity, &s_abort)); };
  uint32_t n_item = 0;       // descriptors this warp has taken
  // the next item's descriptor; false: no more items (or a wait gave up)
  auto next_item = [&](AttnItem& it) -> bool {
    const int slot = n_item % ND;
    if (!wait(B_D_FULL + slot, (n_item / ND) & 1)) return false;
    it = s_item[slot];
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_D_EMPTY + slot));
    ++n_item;
    return it.n_list != 0;
  };

  // Register budget: 640 threads x 96 at launch = 61440 = 256 x 120 (softmax) + 128 x 96 (epilogue) + 256 x 72 (the rest).
  if (warp < W_EPI) {
    // =====================================================================================================
    // softmax groups
    // =====================================================================================================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
    const int g = warp >> 2, row = tid & 127;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tG = tmem + g * 256 + lane_sel, tO = tG + Cfg::COL_O;
    const float scale2 = p.scale * 1.4426950408889634f;
    const bool causal = flash && (p.flags & HA_FLAG_CAUSAL);
    uint32_t buf = 0, par = 0;          // score buffer of the next unit, parity of its barriers
    uint32_t it_g = 0;                  // items this group has taken part in
    bool ok = true;
    HA_T_DECL(8)
    AttnItem it;
    while (ok && next_item(it)) {
      const int n_act = 2 * it.count(g);
      if (n_act == 0) continue;
      const int n_w = 2 * (it.hi(g) - it.lo(g)), lo = 2 * it.lo(g), qt = it.qt0 + g;
      float m_ref = -INFINITY, l_run = 0.f;
#pragma unroll 1
      for (int a = 0; a < n_act; ++a) {
        const int u = a < n_w ? lo + a : 2 * it.n_win + a - n_w;     // unit: half (u & 1) of list entry u / 2
        const uint32_t tS = tG + buf * 64;
        HA_T_MARK(0)
        if (!(ok = wait(B_S_READY + 3 * g + buf, par))) break;
        HA_T_MARK(1)
        tc_fence_after();
        uint32_t s[64];
        {
          uint32_t(&s0)[32] = *reinterpret_cast<uint32_t(*)[32]>(s);
          uint32_t(&s1)[32] = *reinterpret_cast<uint32_t(*)[32]>(s + 32);
          tmem_ld32(tS, s0);
          tmem_ld32(tS + 32, s1);
          tmem_ld_fence(s0);
          tmem_ld_fence(s1);
        }
        // ---- columns this row does not see: past the diagonal, past a ragged last tile, dropped slots of the sample ----
        float bias2 = 0.f;
        if (flash) {
          int limit = p.m_k - u * 64;
          const bool diag = causal && (u >> 1) == qt;
          if (diag) limit = min(limit, row + 1 - (u & 1) * 64);
          if (diag || limit < 64) {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if (i >= limit) s[i] = 0xff800000u;
          }
        } else if (WT && p.sample_logw && u >= 2 * it.n_win) {
          const long long qtile = (long long)it.seg * (p.m_q / TILE) + qt;
          const uint32_t* drop = p.sample_mask + qtile * (p.sample_size / 32) + (u - 2 * it.n_win) * 2;
          const uint32_t d0 = drop[0], d1 = drop[1];
          bias2 = p.sample_logw[qtile] * 1.4426950408889634f;
          if ((d0 | d1) != 0u) {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if (((i < 32 ? d0 : d1) >> (i & 31)) & 1u) s[i] = 0xff800000u;
          }
        }
        float mx;
        {
          float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int i = 0; i < 64; i += 2) m4[(i >> 1) & 3] = fmax3(m4[(i >> 1) & 3], __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
          mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
        }
        const float m_cand = WT ? mx * scale2 + bias2 : mx * scale2;
        const bool move = m_cand > m_ref;
        float alpha = 1.f;
        const bool moved = __any_sync(0xffffffffu, move);
        if (move) {
          alpha = fast_exp2(m_ref - m_cand);
          m_ref = m_cand;
        }
        HA_T_MARK(2)
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        const uint64_t sc2 = pack_f2(scale2, scale2), negm = WT ? pack_f2(bias2 - m_use, bias2 - m_use) : pack_f2(-m_use, -m_use);
        uint64_t ps_a = pack_f2(0.f, 0.f), ps_b = ps_a;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            // of every eight pairs POLY go to the FMA pipe, the others to the exponential unit
            const uint64_t x = ffma2(pack_u2(s[c * 16 + i], s[c * 16 + i + 1]), sc2, negm);
            float p0, p1;
            if ((i >> 1) % 3 == 1 && (i >> 1) / 3 < POLY) {
              poly_exp2_2(x, p0, p1);
            } else {
              unpack_f2(x, p0, p1);
              p0 = fast_exp2(p0);
              p1 = fast_exp2(p1);
            }
            uint64_t& ps = (i & 2) ? ps_b : ps_a;
            ps = fadd2(ps, pack_f2(p0, p1));
            pk[i >> 1] = pack2<T>(p0, p1);
          }
          tmem_st8(tS + c * 8, pk);
        }
        HA_T_MARK(3)
        if (moved && a > 0) {
          // O is complete up to the previous unit: rescale it
          const uint32_t pb = buf == 0 ? NB - 1 : buf - 1;
          if (!(ok = wait(B_PV_DONE + 3 * g + pb, buf == 0 ? par ^ 1 : par))) break;
          tc_fence_after();
          const uint64_t al2 = pack_f2(alpha, alpha);
#pragma unroll 1
          for (int c = 0; c < DV / 64; ++c) {
            uint32_t(&r0)[32] = *reinterpret_cast<uint32_t(*)[32]>(s);
            uint32_t(&r1)[32] = *reinterpret_cast<uint32_t(*)[32]>(s + 32);
            tmem_ld32(tO + c * 64, r0);
            tmem_ld32(tO + c * 64 + 32, r1);
            tmem_ld_fence(r0);
            tmem_ld_fence(r1);
#pragma unroll
            for (int i = 0; i < 64; i += 2) {
              float x, y;
              unpack_f2(fmul2(pack_u2(s[i], s[i + 1]), al2), x, y);
              s[i] = __float_as_uint(x);
              s[i + 1] = __float_as_uint(y);
            }
            tmem_st32(tO + c * 64, r0);
            tmem_st32(tO + c * 64 + 32, r1);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(bar(B_P_READY + 3 * g + buf));
        float s0, s1;
        unpack_f2(fadd2(ps_a, ps_b), s0, s1);
        l_run = l_run * alpha + (s0 + s1);
        if (++buf == NB) { buf = 0; par ^= 1; }
        HA_T_MARK(4)
      }
      if (!ok) break;
      // The epilogue has read the previous item's values (long ago, except where items are a single key tile).
      if (it_g >= 1 && !(ok = wait(B_O_FREE + g, (it_g - 1) & 1))) break;
      s_stat[g * TILE + row] = make_float2(m_ref, l_run);
      mbar_arrive(bar(B_STAT + g));
      ++it_g;
    }
    HA_T_DUMP(8, (int)blockIdx.x * 8, tid == 0)
  } else if (warp < W_S) {
    // =====================================================================================================
    // epilogue group
    // =====================================================================================================
    const int row = tid & 127;
    const uint32_t lane_sel = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t n_out[2] = {0, 0};
    bool ok = true;
    HA_T_DECL(8)
    AttnItem it;
    while (ok && next_item(it)) {
#pragma unroll 1
      for (int g = 0; g < 1 + it.has1; ++g) {
        const int qpos = (it.qt0 + g) * TILE + row;
        int qrow = -1;
        if (qpos < p.m_q) qrow = flash ? qpos : p.q_idx[(long long)it.seg * p.m_q + qpos];
        const long long o_row = (long long)it.q_row0 + (qrow < 0 ? 0 : qrow);
        const long long lse_at = ((long long)(it.b * p.H + it.h)) * p.n + o_row;
        const long long o_at = it.b * p.o_sb + it.h * p.o_sh + o_row * p.o_sn;
        const float lse_old = merge ? p.lse[lse_at] : 0.f;          // requested ahead of the waits
        const uint32_t par = (g ? n_out[1] : n_out[0]) & 1;
        HA_T_MARK(0)
        if (!(ok = wait(B_STAT + g, par) && wait(B_O_FULL + g, par))) break;
        HA_T_MARK(1)
        tc_fence_after();
        const float2 st = s_stat[g * TILE + row];
        const float inv = st.y > 0.f ? 1.f / st.y : 0.f;
        const float lse_own = st.y > 0.f ? (st.x + log2f(st.y)) * 0.6931471805599453f : -INFINITY;
        float lse = lse_own, w1 = 0.f, w2 = 1.f;
        if (merge) {
          const float l1 = lse_old, l2 = lse_own;
          if (p.flags & HA_FLAG_MERGE_EXACT) {
            const float m2 = fmaxf(l1, l2);
            const float e1 = __expf(l1 - m2), e2 = __expf(l2 - m2);
            w1 = e1 / (e1 + e2);
            w2 = e2 / (e1 + e2);
            lse = m2 + __logf(e1 + e2);
          } else {
            const float cf = round_to<T>(1.f / (1.f + __expf(l2 - l1)));
            w1 = cf;
            w2 = round_to<T>(1.f - cf);
            lse = l1 - __logf(cf + 1.1920929e-07f);
          }
        }
        const uint64_t inv2 = pack_f2(inv, inv);
        // 64 columns at a time.  A thread stores its own row, 16 bytes a piece: staging the tile for row-coalesced stores measured
        // no faster.
#pragma unroll 1
        for (int hf = 0; hf < DV / 64; ++hf) {
          uint32_t ra[32], rb[32];
          tmem_ld32(tmem + g * 256 + Cfg::COL_O + lane_sel + hf * 64, ra);
          tmem_ld32(tmem + g * 256 + Cfg::COL_O + lane_sel + hf * 64 + 32, rb);
          tmem_ld_fence(ra);
          tmem_ld_fence(rb);
          if (hf == DV / 64 - 1) {
            tc_fence_before();
            mbar_arrive(bar(B_O_FREE + g));
            HA_T_MARK(2)
          }
          uint32_t w[32];      // the row, normalised and rounded
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float x, y;
            unpack_f2(fmul2(pack_u2(ra[i], ra[i + 1]), inv2), x, y);
            w[i >> 1] = pack2<T>(x, y);
            unpack_f2(fmul2(pack_u2(rb[i], rb[i + 1]), inv2), x, y);
            w[16 + (i >> 1)] = pack2<T>(x, y);
          }
          if (qrow >= 0) {
            if (WT && p.part_o) {      // the un-merged result of this call
              uint4* part = reinterpret_cast<uint4*>((T*)p.part_o + o_at + hf * 64);
#pragma unroll
              for (int e = 0; e < 8; ++e) part[e] = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
            }
            uint4* out = reinterpret_cast<uint4*>((T*)p.o + o_at + hf * 64);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              uint4 v = make_uint4(w[4 * e], w[4 * e + 1], w[4 * e + 2], w[4 * e + 3]);
              if (merge) {
                const uint4 ov = out[e];
                const uint32_t ow[4] = {ov.x, ov.y, ov.z, ov.w}, nw[4] = {v.x, v.y, v.z, v.w};
                uint32_t z[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                  const float2 old = unpack2<T>(ow[h]), mine = unpack2<T>(nw[h]);
                  z[h] = pack2<T>(w1 * old.x + w2 * mine.x, w1 * old.y + w2 * mine.y);
                }
                v = make_uint4(z[0], z[1], z[2], z[3]);
              }
              out[e] = v;
            }
          }
        }
        if (g) ++n_out[1];
        else ++n_out[0];
        if (qrow >= 0) {
          if (WT && p.part_o && p.part_lse) p.part_lse[lse_at] = lse_own;
          p.lse[lse_at] = lse;
        }
        HA_T_MARK(3)
      }
    }
    HA_T_DUMP(8, (int)blockIdx.x * 8 + 5, row == 0)
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp < W_Q) {
      // ===================================================================================================
      // MMA issue, one warp per product and group.  These warps run few instructions between two hand-offs, and every one counts:
      // the chain of a unit passes through them.
      // ===================================================================================================
      constexpr int AB = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
      const int g = warp & 1;
      const uint32_t tG = tmem + g * 256;
      bool ok = true;
      uint32_t slot = warp < W_PV ? 0 : 1, full_par = 0;       // ring slot of the next K (V) tile, parity of its "full" barrier
      uint32_t buf = 0, par = 0;                               // score buffer of the next unit, parity of its barriers
      const bool fence_copies = !(flash && pl.tiles);          // tiles that came by cp.async
      HA_T_DECL(8)
      AttnItem it;
      if (warp < W_PV) {
        // S = Q K^T: 64 keys at a time
        const uint32_t idesc = mma_idesc(TILE, 64, AB, 0, 0);
        uint32_t q_seq = 0;                   // query tiles of the items so far
        bool reused = false;                  // every score buffer has been used once
        while (ok && next_item(it)) {
          const uint32_t qs = q_seq + g, qslot = qs % NQ;
          const uint64_t dQ = smem_desc(s_base + Cfg::OFF_Q + qslot * Cfg::Q_TILE, 16, 1024);
          const bool mine = g == 0 || it.has1;
          const int last = mine ? it.last_entry(g) : -1;
          if (mine) ok = wait(B_Q_FULL + qslot, (qs / NQ) & 1);       // (its fence: the K tile's below)
#pragma unroll 1
          for (int e = 0; e < it.n_list && ok; ++e) {
            HA_T_MARK(0)
            // (waited for by a group the tile is not meant for, too: it may not run ahead of the ring)
            if (!(ok = wait(B_KV_FULL + slot, full_par))) break;
            if (fence_copies) fence_async_smem();
            HA_T_MARK(1)
            if (it.active(g, e)) {
              const uint64_t dK = smem_desc(s_base + Cfg::OFF_KV + slot * Cfg::KV_TILE, 16, 1024);
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                // the product that read P out of this buffer has completed
                if (reused && !(ok = wait(B_PV_DONE + 3 * g + buf, par ^ 1))) break;
                HA_T_MARK(2)
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < D / 16; ++kk) {
                    const uint32_t off = ((kk >> 2) * (TILE * 128) + (kk & 3) * 32) >> 4;
                    mma_ss(tG + buf * 64, dQ + off, dK + off + hf * (8192 >> 4), idesc, kk > 0);
                  }
                  mma_commit(bar(B_S_READY + 3 * g + buf));
                }
                __syncwarp();
                if (++buf == NB) { buf = 0; par ^= 1; reused = true; }
                HA_T_MARK(3)
              }
              if (!ok) break;
            }
            if (elect_one()) {
              mma_commit(bar(B_KV_EMPTY + slot));                    // this group's last read of the tile
              if (e == last) mma_commit(bar(B_Q_EMPTY + qslot));     // ... and of the query tile
            }
            __syncwarp();
            slot += 2;
            if (slot == NKV) { slot = 0; full_par ^= 1; }
            HA_T_MARK(4)
          }
          q_seq += 1 + it.has1;
        }
        HA_T_DUMP(8, (int)blockIdx.x * 8 + 1, lane == 0 && g == 0)
      } else {
        // O += P V
        const uint32_t idesc = mma_idesc(TILE, DV, AB, 0, 1);
        uint32_t n_o = 0;                     // items begun
        while (ok && next_item(it)) {
          const bool mine = g == 0 || it.has1;
          const int first = it.first_entry(g), last = mine ? it.last_entry(g) : -1;
          if (mine) {
            if (n_o >= 1) ok = wait(B_O_FREE + g, (n_o - 1) & 1);      // the previous item's O is out
            ++n_o;
          }
#pragma unroll 1
          for (int e = 0; e < it.n_list && ok; ++e) {
            HA_T_MARK(0)
            if (!(ok = wait(B_KV_FULL + slot, full_par))) break;
            if (fence_copies) fence_async_smem();
            HA_T_MARK(1)
            if (it.active(g, e)) {
              const uint64_t dV = smem_desc(s_base + Cfg::OFF_KV + slot * Cfg::KV_TILE, TILE * 128, 1024);
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                if (!(ok = wait(B_P_READY + 3 * g + buf, par))) break;
                HA_T_MARK(2)
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                  for (int kk = 0; kk < 4; ++kk)
                    mma_ts(tG + Cfg::COL_O, tG + buf * 64 + kk * 8, dV + hf * (8192 >> 4) + kk * (2048 >> 4), idesc, (hf + kk > 0) | (e != first));
                  mma_commit(bar(B_PV_DONE + 3 * g + buf));
                }
                __syncwarp();
                if (++buf == NB) { buf = 0; par ^= 1; }
                HA_T_MARK(3)
              }
              if (!ok) break;
            }
            if (elect_one()) {
              if (e == last) mma_commit(bar(B_O_FULL + g));
              mma_commit(bar(B_KV_EMPTY + slot));                    // this group's last read of the tile
            }
            __syncwarp();
            slot += 2;
            if (slot > NKV) { slot = 1; full_par ^= 1; }
            HA_T_MARK(4)
          }
        }
        HA_T_DUMP(8, (int)blockIdx.x * 8 + 6, lane == 0 && g == 0)
      }
    } else {
      // ===================================================================================================
      // loaders: query tiles, K tiles, V tiles (a warp each for the even and the odd list entries).  The copies of a tile signal its "full"
      // barrier themselves (TMA by their bytes, cp.async by an arrival of every lane), so a loader only waits for free slots and
      // runs ahead across items; the row numbers of its next tile are requested before it waits for this one's slot.
      // The query loader is the scheduler too: it works out the items and publishes their descriptors two items ahead.
      // ===================================================================================================
      const bool is_q = warp == W_Q, is_k = warp == W_K;
      const CUtensorMap* map = &maps.tile[is_q ? 0 : is_k ? 1 : 2];
      const uint16_t* tensor = (const uint16_t*)(is_q ? p.q : is_k ? p.k : p.v);
      const int64_t sb = is_q ? p.q_sb : is_k ? p.k_sb : p.v_sb, sh = is_q ? p.q_sh : is_k ? p.k_sh : p.v_sh, sn = is_q ? p.q_sn : is_k ? p.k_sn : p.v_sn;
      const int slabs = is_q || is_k ? D / 64 : DV / 64;
      const int b_full = is_q ? B_Q_FULL : B_KV_FULL, b_empty = is_q ? B_Q_EMPTY : B_KV_EMPTY;
      const uint32_t ring = is_q ? NQ : NKV;
      const uint32_t s_ring = s_base + (is_q ? Cfg::OFF_Q : Cfg::OFF_KV), s_step = is_q ? Cfg::Q_TILE : Cfg::KV_TILE;
      const int stride = is_q || is_k ? 1 : 2;      // list entries from one tile of this warp to the next
      uint32_t n = is_q || is_k ? 0 : 2 * (warp & 1) + 1;      // ring position of this warp's next tile
      int published = 0;
      auto take = [&](AttnItem& it) -> bool {        // the next item's descriptor; n_list = 0 past the last one
        if (!is_q) return next_item(it);
#pragma unroll 1
        for (; published <= (int)n_item + 2; ++published) {
          const uint32_t slot = published % ND;
          it.n_list = 0;
          const int item = item_of_turn<KIND != FWD_HYPER>(pl, published, blockIdx.x, gridDim.x);
          if (item < pl.n_items) it = attn_item(p, pl, item, flash);
          if (published >= ND && !wait(B_D_EMPTY + slot, (published / ND - 1) & 1)) return false;
          if (lane == 0) {
            s_item[slot] = it;
            mbar_arrive(bar(B_D_FULL + slot));
          }
          __syncwarp();
        }
        it = s_item[n_item % ND];
        ++n_item;
        return it.n_list != 0;
      };
      // indexed tiles by TMA: all of K, and the first query tile -- what is left for the cp.async warps then is a tile each per item
      auto by_gather4 = [&](int e) -> bool { return is_k ? pl.rows & 2 : is_q && e == 0 && (pl.rows & 1); };
      auto row_numbers = [&](const AttnItem& it, int e, int (&rows)[4]) {
        const bool gathered = by_gather4(e);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = gathered ? 4 * lane + q : 32 * q + lane;
          if (is_q) {
            const int pos = (it.qt0 + e) * TILE + r;
            rows[q] = pos >= p.m_q ? -1 : flash ? pos : p.q_idx[(long long)it.seg * p.m_q + pos];
          } else {
            rows[q] = item_key_row(p, it, e, r, flash);
          }
        }
      };
      auto is_boxed = [&](const AttnItem& it, int e) -> bool { return pl.tiles && (flash || (!is_q && e >= it.n_win && !p.sample_idx)); };
      HA_T_DECL(8)
      AttnItem it;
      int e = is_q || is_k ? 0 : warp & 1;
      // moves (it, e) to this warp's next tile; e may lie past the end of the item
      auto settle = [&]() -> bool {
        while (true) {
          const int cnt = is_q ? 1 + it.has1 : it.n_list;
          if (e < cnt) return true;
          e -= cnt;
          if (!take(it)) return false;
        }
      };
      bool more = take(it) && settle();
      int rows[4] = {0, 0, 0, 0};
      if (more && !is_boxed(it, e)) row_numbers(it, e, rows);
      while (more) {
        // this tile
        const bool boxed = is_boxed(it, e), gathered = !boxed && by_gather4(e);
        const int hd = is_q ? it.h : it.hk, b = it.b, row0 = is_q ? it.q_row0 : it.k_row0;
        const int tile0 = row0 + (is_q ? it.qt0 + e : flash ? e : e - it.n_win) * TILE;
        // the next one
        e += stride;
        more = settle();
        int ahead[4] = {0, 0, 0, 0};
        if (more && !is_boxed(it, e)) row_numbers(it, e, ahead);
        const uint32_t slot = n % ring, dst = s_ring + slot * s_step, full = bar(b_full + slot);
        HA_T_MARK(0)
        if (n >= ring && !wait(b_empty + slot, (n / ring - 1) & 1)) break;
        HA_T_MARK(1)
        if (boxed) {
          const int ur = __shfl_sync(0xffffffffu, tile0, 0), uh = __shfl_sync(0xffffffffu, hd, 0), ub = __shfl_sync(0xffffffffu, b, 0);
          if (elect_one()) {
            mbar_expect_tx(full, TILE * 128 * slabs);
#pragma unroll
            for (int s = 0; s < Cfg::W / 64; ++s)
              if (s < slabs) tma_tile(dst + s * TILE * 128, map, s * 64, ur, uh, ub, full);
          } else {
            mbar_arrive(full);
          }
          __syncwarp();
        } else if (gathered) {
          const int x = is_k, step = pl.row_sn[x], base = b * pl.row_sb[x] + hd * pl.row_sh[x] + row0 * step;
          mbar_expect_tx(full, 512 * slabs);     // this lane's four rows
#pragma unroll 1
          for (int s = 0; s < slabs; ++s)
            tma_gather4(dst + s * TILE * 128 + lane * 512, &maps.rows[x], s * 64, base + rows[0] * step, base + rows[1] * step,
                        base + rows[2] * step, base + rows[3] * step, full);
        } else {
          warp_gather_tile(dst, tensor + b * sb + hd * sh + row0 * sn, sn, slabs, rows, lane);
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
        }
        // the next tile's rows into L2 (a copy that finds them there holds its place in the queue for half the time)
        if (!flash && more && !is_boxed(it, e) && (is_q || e < it.n_win)) {
          const uint16_t* base = tensor + it.b * sb + (is_q ? it.h : it.hk) * sh + (int64_t)(is_q ? it.q_row0 : it.k_row0) * sn;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            prefetch_l2(base + (int64_t)ahead[q] * sn);
            if (slabs > 1) prefetch_l2(base + (int64_t)ahead[q] * sn + 64);
          }
        }
        HA_T_MARK(2)
        n += is_q ? 1 : 2 * stride;
#pragma unroll
        for (int q = 0; q < 4; ++q) rows[q] = ahead[q];
      }
      HA_T_DUMP(8, (int)blockIdx.x * 8 + (is_k ? 2 : is_q ? 4 : 3), lane == 0 && (warp <= W_K + 1))
      if (lane == 0) s_issued[warp - W_Q] = n;
      cp_async_commit();
      cp_async_wait<0>();
    }
  }
  // every role is done (or has given up); TMEM goes back
  tc_fence_before();
  __syncthreads();
  if (s_abort) {      // (nobody writes it any more)
    // What is still under way is waited for, with a limit, before TMEM goes and the CTA retires: the last tile of every slot a loader fills,
    // each MMA warp's products, stores to TMEM.  A CTA that gets through its items has waited for all of it on the way.
    const uint32_t bar_end = smem_u32(s_item);      // (the descriptors have been used up: their place takes the MMA warps' barriers)
    if (tid < 4) mbar_init(bar_end + 8 * tid, 1);
    mbar_fence_init();
    __syncthreads();
    if (warp >= W_Q) {
      const uint32_t ring = warp == W_Q ? NQ : NKV, step = warp == W_Q ? 1 : warp == W_K ? 2 : 4, first = warp <= W_K ? 0 : 2 * (warp & 1) + 1;
      const uint32_t n = s_issued[warp - W_Q];
#pragma unroll 1
      for (uint32_t back = step; back <= ring && n >= first + back; back += step)
        mbar_wait(bar((warp == W_Q ? B_Q_FULL : B_KV_FULL) + (n - back) % ring), ((n - back) / ring) & 1);
    } else if (warp >= W_S) {
      mma_settle(bar_end + 8 * (warp - W_S));
    } else {
      tmem_st_wait();
    }
    __syncthreads();
    if (tid == 0) report_timeout(p.status, p.status_host);
  }
  if (warp == W_S) tmem_dealloc(tmem, 512);
}

template <typename T, int D, int DV, int KIND>
static int launch_fwd(const ha_attn_params& p, cudaStream_t st) {
  using Cfg = FwdCfg<D, DV>;
  AttnPlan pl;
  if (!plan_items(pl, p)) return HA_ERR_TOO_LARGE;
  if (pl.n_items == 0) return HA_OK;
  FwdMaps maps;
  const int Hk = p.kv_group > 1 ? p.H / p.kv_group : p.H;
  // rows a head really has on either side (a single-segment call may have fewer or more keys than queries)
  const long long n_q = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.q_off + p.m_q;
  const long long n_k = p.segs_per_head > 1 ? (long long)p.segs_per_head * p.span : p.k_off + p.m_k;
  pl.tiles = boxes_end_with_segments(p) && encode_tile_map(&maps.tile[0], p.dtype, p.q, D, n_q, p.H, p.B, p.q_sn, p.q_sh, p.q_sb, TILE) &&
             encode_tile_map(&maps.tile[1], p.dtype, p.k, D, n_k, Hk, p.B, p.k_sn, p.k_sh, p.k_sb, TILE) &&
             encode_tile_map(&maps.tile[2], p.dtype, p.v, DV, n_k, Hk, p.B, p.v_sn, p.v_sh, p.v_sb, TILE);
  plan_row_maps(pl, p, maps.rows, n_q, n_k);
  // the tiles start at the first 1 KB boundary after the static variables; at head dim 128 they end with the CTA's last byte
  int dyn_bytes;
  HA_WINDOW_BYTES(dyn_bytes, (attn_tc_fwd_kernel<T, D, DV, KIND>), Cfg::SMEM_USED, "ha_attn_fwd kernel attributes");
  HA_SMEM_ATTR_ONCE((attn_tc_fwd_kernel<T, D, DV, KIND>), dyn_bytes, "ha_attn_fwd smem attribute");
  const int sms = sm_count(), grid = pl.n_items < sms ? pl.n_items : sms;
  plan_order(pl, p, grid, 2);
  launch_chained((attn_tc_fwd_kernel<T, D, DV, KIND>), grid, fw::THREADS, dyn_bytes, st, p, pl, maps);
  HA_LAUNCHED("ha_attn_fwd (tcgen05)");
  return HA_OK;
}

bool tc_supported(const ha_attn_params& p) {
  if (p.dtype != HA_BF16 && p.dtype != HA_FP16) return false;
  if (!(p.scale > 0.f)) return false;   // the running max is taken before scaling
  if (!((p.d == 64 || p.d == 128) && (p.dv == 64 || p.dv == 128))) return false;
  // 16-byte row alignment for the copies and vector stores
  auto ok = [](const void* ptr, int64_t sb, int64_t sh, int64_t sn) {
    return ((uintptr_t)ptr % 16 == 0) && sb % 8 == 0 && sh % 8 == 0 && sn % 8 == 0;
  };
  if (!ok(p.q, p.q_sb, p.q_sh, p.q_sn) || !ok(p.k, p.k_sb, p.k_sh, p.k_sn) || !ok(p.v, p.v_sb, p.v_sh, p.v_sn) ||
      !ok(p.o, p.o_sb, p.o_sh, p.o_sn))
    return false;
  if (p.part_o && (uintptr_t)p.part_o % 16 != 0) return false;
  return true;
}

template <typename T>
static int tc_fwd_typed(const ha_attn_params& p, cudaStream_t st) {
  const bool any = (p.flags & HA_FLAG_MERGE) || p.part_o || (p.mode == HA_MODE_HYPER && p.sample_logw && p.sample_size > 0);
#define HA_FWD_CASE(DD, DDV)                                                              \
  if (p.d == DD && p.dv == DDV)                                                           \
    return any ? launch_fwd<T, DD, DDV, FWD_ANY>(p, st)                                   \
               : p.mode == HA_MODE_FLASH ? launch_fwd<T, DD, DDV, FWD_FLASH>(p, st) : launch_fwd<T, DD, DDV, FWD_HYPER>(p, st);
  HA_FWD_CASE(64, 64)
  HA_FWD_CASE(128, 128)
  HA_FWD_CASE(128, 64)
  HA_FWD_CASE(64, 128)
#undef HA_FWD_CASE
  return HA_ERR_INVALID;
}

int tc_attn_fwd(const ha_attn_params& p, cudaStream_t st) {
  return p.dtype == HA_BF16 ? tc_fwd_typed<__nv_bfloat16>(p, st) : tc_fwd_typed<__half>(p, st);
}

}  // namespace ha

HA_T_SETTER(ha_debug_set_timing_buffer_fwd)
